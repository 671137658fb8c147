// Persistent matrix multiply for sm_100a: C[b] = act(A[b] . B[b]^T-layout + add1 + add2) with a dense
// row-major C.  Two operand types, one kernel template: f32 storage with TF32 operands (kind::tf32, 32-element
// K blocks) and f16 storage (kind::f16, 64-element K blocks, f32 accumulation, the result rounded to f16 once in
// the epilogue; an extension, the reference's IR has no half type).  A K block is 128 bytes of either, so
// the pipeline, the shared-memory layout and the operand descriptors are the same.
//
// Compared with the one-tile-per-CTA kernel in contract_tc.cu, a CTA here stays on its SM and walks over
// output tiles, and tensor memory holds TWO accumulators: while the epilogue warps drain tile i
// (tcgen05.ld -> addends / activation -> swizzled staging tile in shared memory -> bulk tensor store),
// the producer is already loading and the MMA thread already multiplying tile i + 1.  For the short-K
// shapes of transformer layers (K = 768: 24 K-blocks per tile) fill and drain were most of a tile's time.
//
//   warp 0, a lane  TMA producer: per K block the 128 x 32 A tile and the BN x 32 B tile (K-major, 128-byte
//                   swizzle, rounded to TF32 by the copy engine), ring of stages with full / empty mbarriers
//   warp 1, a lane  MMA issuer: four tcgen05.mma.kind::tf32 (K = 8) per stage into accumulator `tile & 1`;
//                   waits for that accumulator to be drained, signals it full with tcgen05.commit
//   warps 2..9      epilogue: two groups of four, thread <-> accumulator lane <-> output row; the groups take 32 columns each in
//                   turn; f32 results with nothing added or computed have one (gemm_persistent_prepare).  One group is as fast
//                   while the next tile's MMAs hide it; where a CTA has few tiles or the epilogue adds or computes it is not: 16384 x 768 x 768 + bias 38.8 us with one group and 36.5 with two, 16384 x 3072 x
//                   768 + GELU 136.9 and 129.8, 2048 x 4096 x 4096 of halves 51.9 and 51.3 (without an epilogue to speak of, 2048 x
//                   11008 x 4096 of halves, 129.8 and 130.3).  One warp of a group polls for the accumulator, the rest sleep at
//                   a barrier: with all of them polling, long reductions lost 1% to the power it took.
//
// Large matmuls with a long reduction run on CTA PAIRS (template parameter PAIR, clusters of two): `cta_group::2`
// instructions compute a 256 x BN tile on two SMs, each CTA loading its own 128 rows of A and half of B (see the
// helpers in front of the kernel).  Same instructions in the same K order: results are bit-identical to one CTA per tile.
//
// Tiles are walked column-block-major (all row blocks of one column block before the next), so the CTAs
// that run at the same time share a B tile in L2.  Row and column tails are the copy engine's zero fill
// (loads) and clipping (stores).  Every mbarrier wait is bounded as in the other tensor-core kernels.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>

#include "../tc.h"
#include "tc_host.h"
#include "tc_ptx.cuh"
#include "epilogue.cuh"
#include "launch.cuh"

namespace kn {

namespace {

using namespace tcp;

constexpr int kGpBlockM = 128;
constexpr int kGpBlockK = 32;
constexpr int kGpATileBytes = kGpBlockM * 128;
constexpr int kGpClockTiles = 16;
constexpr int kGpStageTileBytes = 128 * 128;   // epilogue staging: 128 rows x 32 columns of f32

struct GemmPersistentParams {
    int32_t bn, stages, k_iters;
    int32_t groups;           // of epilogue warps, which share two staging tiles
    int32_t a_batch, b_batch;        // 1, or 0 when every batch entry uses the same A / B (batch stride 0)
    int32_t splits, k_iters_slice;   // split K: slice sp of a tile covers K blocks [sp * k_iters_slice, ...) and is stored
                                     // as matrix `batch * splits + sp` of the output map (the partial-sum buffer)
    int32_t m_tiles, n_tiles, batch, total_tiles;
    int64_t m, n;
    const float* add1;
    const float* add2;
    int64_t s1[3], s2[3];            // (batch, row, col) strides of the addends
    int32_t add1_mode, add2_mode;    // 0 absent, 1 one value per column, 2 a value per element (row-contiguous), 4 one value per row
    int32_t act;
    // implicit convolution operand (GemmParams::conv_operand): which operand, 32-channel blocks per filter tap,
    // filter width, padding, output width
    int32_t conv_operand, conv_cblocks, conv_s, conv_pad_y, conv_pad_x, conv_ow;
    // 4-D operands (GemmOperand4D): kd as a shift (0: the K offset is not split), rd, bi; enabled when rd > 0
    int32_t a4_kd_shift, a4_rd, a4_bi, b4_kd_shift, b4_rd, b4_bi;
    int32_t out_half;                // f16 storage and no split: the output tile is f16 (else f32: plain C or partial sums)
    uint32_t* status;
    volatile uint32_t* dbg;          // null, or 8 progress words in pinned host memory (KN_FLAG_TRACE_GEMM)
    long long* clocks;               // KN_GEMM_CLOCKS only: 8 clock64 stamps per tile of CTA 0, in pinned host memory
};

// Post-mortem aid: with KN_FLAG_TRACE_GEMM the first CTA records how far each role got (words: 0 kernel entered,
// 1 K blocks requested, 2 K blocks landed, 3 K blocks multiplied, 4 accumulator seen by the epilogue, 5 chunks
// stored, 6 epilogue done) in pinned host memory, which the host can still read after a fault has taken the
// context.  Off (null pointer) in normal operation.
__device__ __forceinline__ void dbg_mark(const GemmPersistentParams& p, uint32_t slot, uint32_t value) {
    if (p.dbg != nullptr && blockIdx.x == 0) {
        p.dbg[slot] = value;
        __threadfence_system();
    }
}

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_local(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Where the operand tiles of consecutive K blocks lie.  Everything about an operand read in place that does not change
// along K is worked out once per tile, and what does (the filter tap of a K block) is stepped, not divided: the producer's
// loop runs once per K block in ONE thread, and three integer divisions by run-time values in it cost more than the four
// MMAs of the block (measured: a 3x3 convolution over 320 channels ran at 800 cycles per K block instead of 320).
template <bool HALF, bool PAIR>
struct OperandCursor {
    static constexpr int kElems = HALF ? 64 : 32;   // elements per 128-byte K block
    int k, conv_cb = 0, conv_tx = 0, conv_ty = 0, conv_row0 = 0;
    int a4_c1 = 0, a4_c2 = 0, a4_c3 = 0, b4_c1 = 0, b4_c2 = 0, b4_c3 = 0;

    __device__ __forceinline__ OperandCursor(const GemmPersistentParams& p, int a_row0, int b_row0, int bt, int k_begin) : k(k_begin) {
        if (p.conv_operand != 0) {
            const int tap = k_begin / p.conv_cblocks;
            conv_cb = k_begin - tap * p.conv_cblocks;
            conv_ty = tap / p.conv_s;
            conv_tx = tap - conv_ty * p.conv_s;
            conv_row0 = (p.conv_operand == 1 ? a_row0 : b_row0) / p.conv_ow;
        }
        if (p.a4_rd > 0) a4_c1 = a_row0 % p.a4_rd, a4_c2 = bt % p.a4_bi, a4_c3 = a_row0 / p.a4_rd + bt / p.a4_bi;
        if (p.b4_rd > 0) b4_c1 = b_row0 % p.b4_rd, b4_c2 = bt % p.b4_bi, b4_c3 = b_row0 / p.b4_rd + bt / p.b4_bi;
    }
    __device__ __forceinline__ void load3(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) const {
        if (PAIR) tma_load_3d_pair(dst, map, bar, c0, c1, c2);
        else tma_load_3d(dst, map, bar, c0, c1, c2);
    }
    __device__ __forceinline__ void load4(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) const {
        if (PAIR) tma_load_4d_pair(dst, map, bar, c0, c1, c2, c3);
        else tma_load_4d(dst, map, bar, c0, c1, c2, c3);
    }
    // K block k = (filter tap, 32-channel block) of an implicit convolution operand; the tile's rows are whole output rows
    // of image `bt`, so the operand tile is one box of the image tensor (channel, x, y, image) moved by the tap:
    // positions outside the image are the copy engine's zero fill
    __device__ __forceinline__ void load_windows(const GemmPersistentParams& p, const CUtensorMap* map, uint32_t dst, uint32_t bar, int bt) const {
        load4(dst, map, bar, conv_cb * 32, conv_tx - p.conv_pad_x, conv_row0 + conv_ty - p.conv_pad_y, bt);
    }
    // (a head split or merge read in place: the tile's coordinates in the 4-D source, see GemmOperand4D; the row part does
    // not change along K)
    __device__ __forceinline__ void load_a(const GemmPersistentParams& p, const CUtensorMap* map, uint32_t dst, uint32_t bar, int row0, int bt) const {
        const int k0 = k * kElems;
        if (p.conv_operand == 1) {
            load_windows(p, map, dst, bar, bt);
        } else if (p.a4_rd > 0) {
            const int kh = p.a4_kd_shift ? (k0 >> p.a4_kd_shift) : 0;
            load4(dst, map, bar, k0 - (kh << p.a4_kd_shift), a4_c1, kh + a4_c2, a4_c3);
        } else {
            load3(dst, map, bar, k0, row0, bt * p.a_batch);
        }
    }
    __device__ __forceinline__ void load_b(const GemmPersistentParams& p, const CUtensorMap* map, uint32_t dst, uint32_t bar, int row0, int bt) const {
        const int k0 = k * kElems;
        if (p.conv_operand == 2) {
            load_windows(p, map, dst, bar, bt);
        } else if (p.b4_rd > 0) {
            const int kh = p.b4_kd_shift ? (k0 >> p.b4_kd_shift) : 0;
            load4(dst, map, bar, k0 - (kh << p.b4_kd_shift), b4_c1, kh + b4_c2, b4_c3);
        } else {
            load3(dst, map, bar, k0, row0, bt * p.b_batch);
        }
    }
    __device__ __forceinline__ void next(const GemmPersistentParams& p) {
        k++;
        if (p.conv_operand != 0 && ++conv_cb == p.conv_cblocks) {
            conv_cb = 0;
            if (++conv_tx == p.conv_s) { conv_tx = 0; conv_ty++; }
        }
    }
};

// ---- CTA pairs (PAIR): two CTAs of a cluster compute one 256 x BN tile with `cta_group::2` instructions.  Each
// CTA loads its own 128 rows of A and HALF of the B tile; the tensor cores of both SMs read both halves, so every SM's
// shared-memory pipe carries a third fewer bytes per multiply-add than with one CTA per tile (that pipe, not the
// tensor pipe, bounds the one-CTA kernel at about 0.83 of the tensor rate).  CTA 0 of the pair (the leader) issues the
// MMAs; the loads of both CTAs complete on the leader's barriers; `tcgen05.commit` reaches the barriers of both.
// operand storage: f16 (kind::f16) or f32 (kind::tf32); one CTA per tile or a CTA pair; groups of four epilogue warps, which take the
// accumulator's 32-column chunks in turn
template <bool HALF, bool PAIR, int GROUPS>
__global__ void __launch_bounds__(64 + 128 * GROUPS, 1)
gemm_persistent_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_c, const __grid_constant__ GemmPersistentParams p) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int kBlockKElems = HALF ? 64 : 32;   // elements per 128-byte K block
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const int stages = p.stages;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;           // 0: the pair's leader
    const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, n_workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int b_rows = PAIR ? p.bn / 2 : p.bn;                   // rows of the B tile this CTA loads
    const uint32_t b_tile_bytes = (uint32_t)b_rows * 128u;
    const uint32_t stage_bytes = kGpATileBytes + b_tile_bytes;
    const uint32_t staging_base = base + (uint32_t)stages * stage_bytes;          // two staging tiles
    const uint32_t bar_base = staging_base + 2u * kGpStageTileBytes;
    const uint32_t full_bar = bar_base, empty_bar = bar_base + 8u * stages;
    const uint32_t acc_full = bar_base + 16u * stages, acc_empty = acc_full + 16u;
    const uint32_t slot_addr = acc_empty + 16u;
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + (slot_addr - base));
    volatile int* abandon = (volatile int*)(gen_base + (slot_addr + 4u - base));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(full_bar + 8u * s, 1);
            mbar_init(empty_bar + 8u * s, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full + 8u * b, 1);
            mbar_init(acc_empty + 8u * b, (PAIR ? 8 : 4) * GROUPS);   // (a warp each; pair: those of both CTAs arrive on the leader's)
        }
        *abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (PAIR) cluster_sync_all();   // the peer's barriers are initialised before anything is sent to them
    const uint32_t tmem_cols = 2u * (uint32_t)p.bn <= 32u ? 32u : (2u * (uint32_t)p.bn <= 64u ? 64u : (2u * (uint32_t)p.bn <= 128u ? 128u : (2u * (uint32_t)p.bn <= 256u ? 256u : 512u)));
    if (warp == 0) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // nothing above touches global memory

    // tile t -> (row block, column block, batch): row blocks fastest
    auto tile_coords = [&](int t, int& mt, int& nt, int& bt, int& sp) {
        mt = t % p.m_tiles;
        const int r = t / p.m_tiles;
        nt = r % p.n_tiles;
        const int r2 = r / p.n_tiles;
        sp = r2 % p.splits;
        bt = r2 / p.splits;
    };
    auto slice_blocks = [&](int sp) { return min(p.k_iters_slice, p.k_iters - sp * p.k_iters_slice); };

    if (threadIdx.x == 0) dbg_mark(p, 0, 1);
    if (warp == 0 && elect_one()) {
        // ---------------- producer
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        int s = 0, round = 0;
        bool ok = true;
        for (int t = worker; t < p.total_tiles && ok; t += n_workers) {
            int mt, nt, bt, sp;
            tile_coords(t, mt, nt, bt, sp);
            const int k_begin = sp * p.k_iters_slice, k_end = k_begin + slice_blocks(sp);
            const int a_row0 = (PAIR ? 2 * mt + (int)rank : mt) * kGpBlockM;   // this CTA's rows of A
            const int b_row0 = nt * p.bn + (PAIR ? (int)rank * b_rows : 0);      // and of B (a pair: its half)
            OperandCursor<HALF, PAIR> cursor(p, a_row0, b_row0, bt, k_begin);
            for (int k = k_begin; k < k_end; k++) {
                if (round > 0 && !mbar_wait(empty_bar + 8u * s, (uint32_t)((round & 1) ^ 1), abandon, p.status, 21)) { ok = false; break; }
                const uint32_t bar = full_bar + 8u * s;
                const uint32_t dst = base + (uint32_t)s * stage_bytes;
                // pair: both CTAs' tiles complete on the LEADER's barrier, which expects the bytes of both
                if (!PAIR || rank == 0) mbar_expect_tx(bar, PAIR ? 2u * stage_bytes : stage_bytes);
                const uint32_t to_bar = PAIR ? map_to_cta(bar, 0) : bar;
                cursor.load_a(p, &map_a, dst, to_bar, a_row0, bt);
                cursor.load_b(p, &map_b, dst + kGpATileBytes, to_bar, b_row0, bt);
                cursor.next(p);
                dbg_mark(p, 1, (uint32_t)(k + 1));
                if (++s == stages) { s = 0; round++; }
            }
        }
    } else if (PAIR && warp == 1 && rank != 0) {
        // the peer issues no MMAs (the leader's instructions drive both tensor cores)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    } else if (warp == 1 && elect_one()) {
        // ---------------- MMA issuer
        // instruction descriptor: f32 accumulate; A and B formats 2 = TF32 (kind::tf32) or 0 = F16 (kind::f16); both
        // K-major; N, M
        const uint32_t fmt = HALF ? 0u : 2u;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.bn >> 3) << 17) |
                               ((uint32_t)((PAIR ? 2 * kGpBlockM : kGpBlockM) >> 4) << 24);
        int s = 0, round = 0, local = 0;
        bool ok = true;
        for (int t = worker; t < p.total_tiles && ok; t += n_workers, local++) {
            const int buf = local & 1;
            const bool clk = p.clocks != nullptr && blockIdx.x == 0 && local < kGpClockTiles;
            if (clk) p.clocks[local * 8 + 0] = clock64();
            // the epilogue has drained this accumulator (its previous use was tile local - 2)
            if (local >= 2 && !mbar_wait(acc_empty + 8u * buf, (uint32_t)(((local >> 1) - 1) & 1), abandon, p.status, 22)) break;
            tc_fence_after();
            if (clk) p.clocks[local * 8 + 1] = clock64();
            const uint32_t acc = tmem_base + (uint32_t)(buf * p.bn);
            int mt, nt, bt, sp;
            tile_coords(t, mt, nt, bt, sp);
            const int k_count = slice_blocks(sp);
            // last tile of this CTA: the next kernel of the stream may be scheduled (once every CTA says so)
            if (t + n_workers >= p.total_tiles) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            for (int k = 0; k < k_count; k++) {
                if (!mbar_wait(full_bar + 8u * s, (uint32_t)(round & 1), abandon, p.status, 23)) { ok = false; break; }
                if (clk && k == 0) p.clocks[local * 8 + 2] = clock64();
                dbg_mark(p, 2, (uint32_t)(k + 1));
                tc_fence_after();
                const uint32_t a_addr = base + (uint32_t)s * stage_bytes;
                const uint64_t da = smem_desc_sw128(a_addr);
                const uint64_t db = smem_desc_sw128(a_addr + kGpATileBytes);
                // four instructions of 32 bytes of K each: the start address advances by 2 (16-byte units)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (PAIR) mma_pair<HALF>(acc, da + 2u * j, db + 2u * j, idesc, (k | j) != 0 ? 1u : 0u);
                    else if (HALF) mma_f16(acc, da + 2u * j, db + 2u * j, idesc, (k | j) != 0 ? 1u : 0u);
                    else mma_tf32(acc, da + 2u * j, db + 2u * j, idesc, (k | j) != 0 ? 1u : 0u);
                }
                if (PAIR) mma_commit_pair(empty_bar + 8u * s);
                else mma_commit(empty_bar + 8u * s);
                dbg_mark(p, 3, (uint32_t)(k + 1));
                if (++s == stages) { s = 0; round++; }
            }
            if (ok) {
                if (PAIR) mma_commit_pair(acc_full + 8u * buf);
                else mma_commit(acc_full + 8u * buf);
                if (clk) p.clocks[local * 8 + 3] = clock64();
            }
        }
    } else if (warp >= 2) {
        // ---------------- epilogue
        const int quarter = warp & 3;
        const int row_in_tile = quarter * 32 + lane;
        const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
        const int group = GROUPS == 1 ? 0 : (warp - 2) >> 2;   // of two: has chunks group, group + 2, ... and a staging tile of its own
        const bool issuer = ((threadIdx.x - 64) & 127) == 0;   // the thread of the group that talks to the copy engine
        // swizzled position of this row's 16-byte chunk c inside a staging tile: chunk ^ (row & 7)
        const uint32_t row_base = (uint32_t)row_in_tile * 128u;
        const uint32_t row_phase = (uint32_t)row_in_tile & 7u;
        int local = 0;
        bool ok = true;
        auto group_sync = [&]() {   // (of a barrier that the instruction names: one from a register takes longer)
            if (group == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
            else asm volatile("bar.sync 2, 128;" ::: "memory");
        };
        uint32_t staging = staging_base + (uint32_t)group * kGpStageTileBytes;
        for (int t = worker; t < p.total_tiles && ok; t += n_workers, local++) {
            int mt, nt, bt, sp;
            tile_coords(t, mt, nt, bt, sp);
            if (PAIR) mt = 2 * mt + (int)rank;   // from here on: this CTA's 128-row block
            const int buf = local & 1;
            {
                uint32_t good = 1;
                if (lane == 0 && (warp - 2) % 4 == 0) good = mbar_wait(acc_full + 8u * buf, (uint32_t)((local >> 1) & 1), abandon, p.status, 24) ? 1u : 0u;
                good = __shfl_sync(0xffffffffu, good, 0);
                // the loop below synchronises the group's four warps with each other, so they must agree on
                // entering it: vote (every epilogue thread gets here, its wait being bounded)
                uint32_t all_good;
                if (group == 0)
                    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 3, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(all_good) : "r"(good) : "memory");
                else
                    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 4, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(all_good) : "r"(good) : "memory");
                if (!all_good) { ok = false; break; }
                while (!mbar_try_wait(acc_full + 8u * buf, (uint32_t)((local >> 1) & 1))) {}
            }
            tc_fence_after();
            const bool eclk = p.clocks != nullptr && blockIdx.x == 0 && local < kGpClockTiles && threadIdx.x == 64;
            long long store_wait = 0;
            if (eclk) p.clocks[local * 8 + 4] = clock64();
            if (issuer) dbg_mark(p, 4, 1);
            const int64_t row = (int64_t)mt * kGpBlockM + row_in_tile;
            const bool row_ok = row < p.m;
            const int chunks = (p.bn + 31) >> 5;
            for (int c = group; c < chunks; c += GROUPS) {
                const int col0 = nt * p.bn + c * 32;
                if (col0 >= p.n) break;                       // uniform: nothing of this chunk is inside the matrix
                uint32_t v[32];
                tmem_load_32(tmem_base + lane_bits + (uint32_t)(buf * p.bn + c * 32), v);
                // addends: a per-column value is fetched once per chunk (lane j holds column col0 + j) and
                // handed round with shuffles; a per-element addend is this thread's own row, 128 contiguous bytes
#pragma unroll
                for (int which = 0; which < 2; which++) {
                    const int mode = which == 0 ? p.add1_mode : p.add2_mode;
                    if (mode == 0) continue;
                    const float* add = which == 0 ? p.add1 : p.add2;
                    const int64_t* st = which == 0 ? p.s1 : p.s2;
                    if (HALF) {
                        // f16 addends: converted on load
                        const __half* addh = (const __half*)add;
                        if (mode == 1) {
                            const int64_t col = col0 + lane;
                            const float mine = col < p.n ? __half2float(__ldg(addh + bt * st[0] + col * st[2])) : 0.f;
#pragma unroll
                            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __shfl_sync(0xffffffffu, mine, j));
                        } else if (mode == 4) {
                            const float mine = row_ok ? __half2float(__ldg(addh + bt * st[0] + row * st[1])) : 0.f;
#pragma unroll
                            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + mine);
                        } else if (row_ok) {
                            const __half* src = addh + bt * st[0] + row * st[1] + col0;
                            if (col0 + 32 <= p.n && ((uintptr_t)src & 15) == 0) {
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const uint4 a8 = __ldg((const uint4*)src + q);
                                    const __half2* h2 = (const __half2*)&a8;
#pragma unroll
                                    for (int u = 0; u < 4; u++) {
                                        const float2 f = __half22float2(h2[u]);
                                        v[8 * q + 2 * u] = __float_as_uint(__uint_as_float(v[8 * q + 2 * u]) + f.x);
                                        v[8 * q + 2 * u + 1] = __float_as_uint(__uint_as_float(v[8 * q + 2 * u + 1]) + f.y);
                                    }
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; j++)
                                    if (col0 + j < p.n) v[j] = __float_as_uint(__uint_as_float(v[j]) + __half2float(__ldg(src + j)));
                            }
                        }
                        continue;
                    }
                    const float* cols = add + bt * st[0] + (int64_t)col0 * st[2];
                    if (mode == 1 && st[2] == 1 && col0 + 32 <= p.n && ((uintptr_t)cols & 15) == 0) {
                        // (every lane reads the same 128 bytes; a shuffle per column takes four times as long)
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const float4 a4 = __ldg((const float4*)cols + q);
                            v[4 * q] = __float_as_uint(__uint_as_float(v[4 * q]) + a4.x);
                            v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + a4.y);
                            v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + a4.z);
                            v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + a4.w);
                        }
                    } else if (mode == 1) {
                        const int64_t col = col0 + lane;
                        const float mine = col < p.n ? __ldg(add + bt * st[0] + col * st[2]) : 0.f;
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __shfl_sync(0xffffffffu, mine, j));
                    } else if (mode == 4) {
                        const float mine = row_ok ? __ldg(add + bt * st[0] + row * st[1]) : 0.f;
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + mine);
                    } else if (row_ok) {
                        const float* src = add + bt * st[0] + row * st[1] + col0;
                        if (col0 + 32 <= p.n && ((uintptr_t)src & 15) == 0) {
#pragma unroll
                            for (int q = 0; q < 8; q++) {
                                const float4 a4 = __ldg((const float4*)src + q);
                                v[4 * q] = __float_as_uint(__uint_as_float(v[4 * q]) + a4.x);
                                v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + a4.y);
                                v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + a4.z);
                                v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + a4.w);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (col0 + j < p.n) v[j] = __float_as_uint(__uint_as_float(v[j]) + __ldg(src + j));
                        }
                    }
                }
                if (p.act == (int)Activation::Relu) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __float_as_uint(fmaxf(__uint_as_float(v[j]), 0.f));
                } else if (p.act == (int)Activation::Gelu) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __float_as_uint(gelu_erf_tensor_core(__uint_as_float(v[j])));
                }
                // the staging tile about to be written was handed to the copy engine with the group's last chunk, or the one before
                if (issuer) {
                    const long long t0 = eclk ? clock64() : 0;
                    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(GROUPS == 1 ? 1 : 0) : "memory");
                    if (eclk) store_wait += clock64() - t0;
                }
                group_sync();
                if (HALF && p.out_half) {
                    // f16 output: rows of 32 halves = 64 bytes, plain row-major (the store map has no swizzle)
                    const uint32_t stile = staging + (uint32_t)row_in_tile * 64u;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        uint32_t h[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const __half2 pair = __floats2half2_rn(__uint_as_float(v[8 * q + 2 * u]), __uint_as_float(v[8 * q + 2 * u + 1]));
                            h[u] = *(const uint32_t*)&pair;
                        }
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stile + (uint32_t)q * 16u), "r"(h[0]), "r"(h[1]),
                                     "r"(h[2]), "r"(h[3])
                                     : "memory");
                    }
                } else {
                    const uint32_t stile = staging + row_base;
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stile + (((uint32_t)q ^ row_phase) << 4)),
                                     "r"(v[4 * q]), "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3])
                                     : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                group_sync();
                if (issuer) {
                    tma_store_3d(&map_c, staging, col0, mt * kGpBlockM, bt * p.splits + sp);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    dbg_mark(p, 5, (uint32_t)(c + 1));
                }
                if (GROUPS == 1) staging = staging == staging_base ? staging_base + kGpStageTileBytes : staging_base;
            }
            if (eclk) p.clocks[local * 8 + 5] = clock64(), p.clocks[local * 8 + 6] = store_wait;
            // every tcgen05.ld of this accumulator has completed (tmem_load_32 waits): the MMA thread may reuse it
            // (the arrival hands over nothing in memory: no release at cluster scope, which waits for all of a thread's stores)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_remote(map_to_cta(acc_empty + 8u * buf, 0));
                else mbar_arrive_local(acc_empty + 8u * buf);
            }
        }
        if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory must outlive the stores
        if (issuer) dbg_mark(p, 6, 1);
    }

    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still address it
    if (warp == 0) {
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ---- Few tiles: a matmul of less than one round of 128 x 256 tiles (a short prompt or sentence, a small image, the last
// layers of a head).  One tile and one slice of K per CTA; the slices of a tile are a CLUSTER, which sums the partial tiles
// through distributed shared memory, so there is neither a scratch buffer in global memory nor a second kernel.  What
// bounds these shapes is how soon and how fast the operands reach shared memory, hence:
//   - narrower tiles and slices of K until the chip has a CTA per SM (gemm_slices_choose weighs the bytes per CTA),
//   - an operand that is a constant (the weights) is requested BEFORE `griddepcontrol.wait`, under the previous kernel's
//     tail, as many K blocks of it as there are stages,
//   - the next kernel is released at once, so that it can do the same.
// The partial tile goes to shared memory (row pitch bn + 4 floats: conflict-free for 16-byte accesses), CTA r of the
// cluster sums rows [r * per, (r + 1) * per) in slice order, adds the addends and stores along the rows; any strides, any
// alignment.  Stored rows are bound by instructions (eight epilogue warps, each address and predicate counts) and, with
// slices, by the 16 bytes per cycle that an SM reads from other SMs' shared memory.  Hence four columns of a fixed column
// group per thread, rows a constant step apart, variants of the loop by addends and slices, and addends that differ by row
// requested four rows ahead, the first of them under the MMAs.  (Item by item, with addresses, addends and predicates worked
// out for each, a tile's way out took 5 000 to 25 000 of the kernel's 20 000 to 60 000 cycles; sent as 16-byte remote stores
// instead of read, the partial sums of four slices and more took half as long again.)
// The producer's and the issuer's warps are not epilogue warps: set-up of the epilogue would otherwise follow the last MMA.
// At most 96 registers a thread: two CTAs to an SM, this kernel's and the next one's among them.  The f32 loops over rows with two
// addends that differ by row do not fit that (104 bytes of stack, nearly all of it theirs).
// us a launch, before the epilogue by column groups -> now: 120 x 2304 x 768 9.7 -> 8.4, 120 x 3072 x 768 + GELU 10.8 -> 10.3,
// 333 x 4096 x 4096 f16 21.0 -> 17.2, 333 x 4096 x 11008 f16 38.6 -> 36.0, 333 x 11008 x 4096 f16 40.4 -> 33.3,
// 4096 x 320 x 320 + bias + skip 16.6 -> 8.0, 4096 x 320 x 1280 + bias + skip 21.8 -> 13.9, 3x3 convolution of 32 x 32
// positions, 640 -> 640 channels 26.4 -> 24.0.
constexpr int kGsThreads = 320;   // eight epilogue warps, the producer's and the issuer's
constexpr int kGsEpilogue = 256;
constexpr int kGsMaxSlices = 8;   // the largest portable cluster
constexpr int kGsBatch = 4;       // rows that a thread of the epilogue has in flight

struct GemmSlicesParams {
    GemmPersistentParams g;
    void* out;
    int64_t so[3];
    int32_t a_const, b_const;                 // the operand is a constant
    int32_t out_vec, add1_vec, add2_vec;      // rows contiguous, every row start aligned to four elements
    int32_t tmem_cols;
};

__device__ __forceinline__ void add_four(float (&v)[4], const float* src, int64_t col_stride, bool vec, int valid) {
    if (vec && valid == 4) {
        const float4 a = *(const float4*)src;
        v[0] += a.x, v[1] += a.y, v[2] += a.z, v[3] += a.w;
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (j < valid) v[j] += src[j * col_stride];
}

template <bool HALF>
__global__ void __launch_bounds__(kGsThreads, 2)
gemm_slices_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ GemmSlicesParams q) {
    extern __shared__ uint8_t smem_raw[];
    const GemmPersistentParams& p = q.g;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const int stages = p.stages;
    const uint32_t stage_bytes = kGpATileBytes + (uint32_t)p.bn * 128u;
    const uint32_t pitch = (uint32_t)(p.bn + 4) * 4u;
    const uint32_t bar_base = base + max((uint32_t)stages * stage_bytes, (uint32_t)kGpBlockM * pitch);
    const uint32_t full_bar = bar_base, empty_bar = bar_base + 8u * stages, acc_full = bar_base + 16u * stages;
    const uint32_t slot_addr = acc_full + 8u;
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + (slot_addr - base));
    volatile int* abandon = (volatile int*)(gen_base + (slot_addr + 4u - base));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(full_bar + 8u * s, 1);
            mbar_init(empty_bar + 8u * s, 1);
        }
        mbar_init(acc_full, 1);
        *abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"((uint32_t)q.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // (after the allocation of tensor memory: a CTA of the next kernel that takes its own first would keep this one waiting)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int splits = p.splits;
    const int sp = (int)(blockIdx.x % (unsigned)splits), t = (int)(blockIdx.x / (unsigned)splits);   // sp: rank in the cluster
    const int mt = t % p.m_tiles, r = t / p.m_tiles, nt = r % p.n_tiles, bt = r / p.n_tiles;
    const int k_begin = sp * p.k_iters_slice, k_count = min(p.k_iters_slice, p.k_iters - k_begin);
    const int a_row0 = mt * kGpBlockM, b_row0 = nt * p.bn;

    bool good = true;
    if (warp == 8) {
        // ---------------- producer.  Lane s fills stage s first: one pass over the set-up arithmetic for all stages (stage by
        // stage in one thread, launches of 120 rows took 5 to 20 % longer)
        const int first = min(stages, k_count);
        {
            const OperandCursor<HALF, false> cursor(p, a_row0, b_row0, bt, k_begin + lane);
            const uint32_t dst = base + (uint32_t)lane * stage_bytes, bar = full_bar + 8u * lane;
#pragma unroll 1
            for (int pass = 0; pass < 2; pass++) {   // the constant operand, then the other
                if (pass == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
                if (lane < first) {
                    if (pass == 0) mbar_expect_tx(bar, stage_bytes);
                    if ((q.a_const != 0) == (pass == 0)) cursor.load_a(p, &map_a, dst, bar, a_row0, bt);
                    if ((q.b_const != 0) == (pass == 0)) cursor.load_b(p, &map_b, dst + kGpATileBytes, bar, b_row0, bt);
                }
            }
        }
        if (k_count > first && elect_one()) {
            OperandCursor<HALF, false> cursor(p, a_row0, b_row0, bt, k_begin + first);
            int s = 0, round = 1;
#pragma unroll 1
            for (int k = first; k < k_count; k++) {
                if (!mbar_wait(empty_bar + 8u * s, (uint32_t)((round & 1) ^ 1), abandon, p.status, 31)) break;
                const uint32_t dst = base + (uint32_t)s * stage_bytes, bar = full_bar + 8u * s;
                mbar_expect_tx(bar, stage_bytes);
                cursor.load_a(p, &map_a, dst, bar, a_row0, bt);
                cursor.load_b(p, &map_b, dst + kGpATileBytes, bar, b_row0, bt);
                cursor.next(p);
                if (++s == stages) { s = 0; round++; }
            }
        }
    } else if (warp == 9 && elect_one()) {
        // ---------------- MMA issuer (the instruction descriptor of gemm_persistent_kernel)
        // (the clock of a bounded wait starts when the kernels in front are done, however long they take)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t fmt = HALF ? 0u : 2u;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(kGpBlockM >> 4) << 24);
        int s = 0, round = 0;
        for (int k = 0; k < k_count && good; k++) {
            if (!mbar_wait(full_bar + 8u * s, (uint32_t)(round & 1), abandon, p.status, 32)) { good = false; break; }
            tc_fence_after();
            const uint32_t a_addr = base + (uint32_t)s * stage_bytes;
            const uint64_t da = smem_desc_sw128(a_addr), db = smem_desc_sw128(a_addr + kGpATileBytes);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (HALF) mma_f16(tmem_base, da + 2u * j, db + 2u * j, idesc, (k | j) != 0 ? 1u : 0u);
                else mma_tf32(tmem_base, da + 2u * j, db + 2u * j, idesc, (k | j) != 0 ? 1u : 0u);
            }
            mma_commit(empty_bar + 8u * s);
            if (++s == stages) { s = 0; round++; }
        }
        if (good) mma_commit(acc_full);
    }
    __syncwarp();

    // The result's rows of this CTA: a thread of the epilogue takes four columns of every row_step-th row
    const int rows = (int)min((int64_t)kGpBlockM, p.m - (int64_t)mt * kGpBlockM), per = (rows + splits - 1) / splits;
    const int my_rows = max(0, min(per, rows - sp * per));
    const int cols = (int)min((int64_t)p.bn, p.n - (int64_t)nt * p.bn), groups = (cols + 3) >> 2;
    const int row_step = kGsEpilogue / groups, row0 = threadIdx.x / groups, col = (threadIdx.x - row0 * groups) * 4, valid = min(4, cols - col);
    const bool mine = row0 < row_step;
    using T = typename std::conditional<HALF, __half, float>::type;
    auto whole = [&](const float* addend, const int64_t* st, bool aligned) { return addend == nullptr || aligned || st[2] == 0; };
    const bool vec = q.out_vec != 0 && (cols & 3) == 0 && whole(p.add1, p.s1, q.add1_vec) && whole(p.add2, p.s2, q.add2_vec);
    // An addend that all rows share is read once, any other a batch of rows ahead (the first batch under the MMAs), as
    // `extra` and, if there are two, `extra2`
    const bool rows1 = p.add1 && p.s1[1] != 0, rows2 = p.add2 && p.s2[1] != 0;
    const int extras = (rows1 ? 1 : 0) + (rows2 ? 1 : 0);   // (results of f16 have no addends: the sum would round once more)
    const float *add1 = nullptr, *add2 = nullptr, *extra = nullptr, *extra2 = nullptr;
    const int64_t extra_row = rows1 ? p.s1[1] : p.s2[1], extra2_row = p.s2[1];
    const bool extra_one = (rows1 ? p.s1[2] : p.s2[2]) == 0, extra2_one = p.s2[2] == 0;   // one value per row
    T* out = nullptr;
    float shared[4] = {0.f, 0.f, 0.f, 0.f};
    float4 next[kGsBatch], next2[kGsBatch];
    auto four = [&](const float* from, bool one) { return one ? make_float4(*from, *from, *from, *from) : *(const float4*)from; };
    auto fetch = [&](int row) {
#pragma unroll
        for (int i = 0; i < kGsBatch; i++) {
            const int r = row + i * row_step;
            if (r < my_rows) {
                next[i] = four(extra + r * extra_row, extra_one);
                if (extras > 1) next2[i] = four(extra2 + r * extra2_row, extra2_one);
            }
        }
    };
    if (warp < kGsEpilogue / 32) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (the addends and the output belong to earlier kernels until here)
        const int64_t m = (int64_t)mt * kGpBlockM + sp * per, n = (int64_t)nt * p.bn + col;
        out = (T*)q.out + bt * q.so[0] + m * q.so[1] + n * q.so[2];
        if (p.add1) add1 = p.add1 + bt * p.s1[0] + m * p.s1[1] + n * p.s1[2];
        if (p.add2) add2 = p.add2 + bt * p.s2[0] + m * p.s2[1] + n * p.s2[2];
        extra = rows1 ? add1 : add2, extra2 = add2;
        if (mine && vec) {
            if (p.add1 && !rows1) add_four(shared, add1, p.s1[2], q.add1_vec != 0, 4);
            if (p.add2 && !rows2) add_four(shared, add2, p.s2[2], q.add2_vec != 0, 4);
            if (extras) fetch(row0);
        }
        // the accumulator is complete, and with it every read of the stages: they become the partial tile
        if (lane == 0) good = mbar_wait(acc_full, 0, abandon, p.status, 33, kWaitCycles, 1000) && good;
    }
    good = __syncthreads_and(good ? 1 : 0) != 0;
    if (good && warp < kGsEpilogue / 32) {
        tc_fence_after();
        const int quarter = warp & 3;
        const uint32_t row_addr = base + (uint32_t)(quarter * 32 + lane) * pitch;
#pragma unroll 1
        for (int c = warp >> 2; c < (p.bn >> 5); c += kGsEpilogue / 128) {
            uint32_t v[32];
            tmem_load_32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 32), v);
#pragma unroll
            for (int j = 0; j < 8; j++)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + (uint32_t)(c * 128 + j * 16)), "r"(v[4 * j]),
                             "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                             : "memory");
        }
        tc_fence_before();
    }
    if (splits > 1) cluster_sync_all();   // every slice's partial tile lies in its CTA's shared memory
    else __syncthreads();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)q.tmem_cols) : "memory");

    auto activate = [&](float (&y)[4]) {
#pragma unroll 1
        for (int j = 0; j < 4; j++) {   // (rolled: the error function would be most of the epilogue's code)
            const float t = apply_activation(y[0], p.act);
            y[0] = y[1], y[1] = y[2], y[2] = y[3], y[3] = t;
        }
    };
    // four columns of a row of a slice's partial tile, from this CTA's rows on
    const uint32_t from = base + (uint32_t)(sp * per) * pitch + (uint32_t)col * 4u;
    auto partial = [&](float (&x)[4], uint32_t at) {
        if (splits == 1) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(at));
        else asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(at));
    };
    const int end = good && mine && warp < kGsEpilogue / 32 ? my_rows : 0;
    // kGsBatch rows at a time, with eight reads of partial sums in flight: of S slices and the rows that leaves.  What this
    // loop costs is instructions (two warps a scheduler), so what does not change in it is decided outside
    auto store_rows = [&](auto most, auto added) {
        constexpr int S = decltype(most)::value, R = S == 1 ? kGsBatch : 8 / S, EXTRAS = decltype(added)::value;
        uint32_t peer[S];
#pragma unroll
        for (int s = 0; s < S; s++) peer[s] = S == 1 ? from : map_to_cta(from, (uint32_t)min(s, splits - 1));
#pragma unroll 1
        for (int row = row0; row < end; row += kGsBatch * row_step) {
            float y[kGsBatch][4];
            bool in[kGsBatch];
#pragma unroll
            for (int i = 0; i < kGsBatch; i++) in[i] = row + i * row_step < end;
#pragma unroll
            for (int i = 0; i < kGsBatch; i += R) {
                if (i > 0 && !in[i]) break;   // (few rows a thread: eight slices of 134 x 32 results 5.9 -> 5.6 us, 5.6 before there were batches)
                float x[R][S][4];
#pragma unroll
                for (int r = 0; r < R; r++) {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (in[i + r] && (S <= 2 || s < splits)) partial(x[r][s], peer[s] + (uint32_t)(row + (i + r) * row_step) * pitch);
                }
#pragma unroll
                for (int r = 0; r < R; r++) {
#pragma unroll
                    for (int j = 0; j < 4; j++) y[i + r][j] = x[r][0][j];
#pragma unroll
                    for (int s = 1; s < S; s++) {
                        if (S > 2 && s >= splits) break;
#pragma unroll
                        for (int j = 0; j < 4; j++) y[i + r][j] += x[r][s][j];
                    }
                }
                if constexpr (S == 4) {
#pragma unroll 1
                    for (int s = S; s < splits; s++) {   // (of more than four slices, with two addends: no registers for eight)
#pragma unroll
                        for (int r = 0; r < R; r++)
                            if (in[i + r]) partial(x[r][0], map_to_cta(from, (uint32_t)s) + (uint32_t)(row + (i + r) * row_step) * pitch);
#pragma unroll
                        for (int r = 0; r < R; r++) {
#pragma unroll
                            for (int j = 0; j < 4; j++) y[i + r][j] += x[r][0][j];
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kGsBatch; i++) {
                auto add = [&](const float4& a) { y[i][0] += a.x, y[i][1] += a.y, y[i][2] += a.z, y[i][3] += a.w; };
#pragma unroll
                for (int j = 0; j < 4; j++) y[i][j] += shared[j];
                if constexpr (EXTRAS > 0) add(next[i]);
                if constexpr (EXTRAS > 1) add(next2[i]);
            }
            if constexpr (EXTRAS > 0) fetch(row + kGsBatch * row_step);
            if (p.act == (int)Activation::Relu) {
#pragma unroll
                for (int i = 0; i < kGsBatch; i++) {
#pragma unroll
                    for (int j = 0; j < 4; j++) y[i][j] = fmaxf(y[i][j], 0.f);
                }
            } else if (p.act != (int)Activation::None) {
#pragma unroll
                for (int i = 0; i < kGsBatch; i++)
                    if (in[i]) activate(y[i]);
            }
            T* dst = out + (int64_t)row * q.so[1];
#pragma unroll
            for (int i = 0; i < kGsBatch; i++, dst += (int64_t)row_step * q.so[1]) {
                if (!in[i]) continue;
                if constexpr (HALF) {
                    const __half2 lo = __floats2half2_rn(y[i][0], y[i][1]), hi = __floats2half2_rn(y[i][2], y[i][3]);
                    *(uint2*)dst = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
                } else {
                    *(float4*)dst = make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
                }
            }
        }
    };
    auto store_all = [&](auto most) {
        if constexpr (HALF) store_rows(most, std::integral_constant<int, 0>());
        else if (extras == 0) store_rows(most, std::integral_constant<int, 0>());
        else if (extras == 1) store_rows(most, std::integral_constant<int, 1>());
        else if constexpr (decltype(most)::value <= 4) store_rows(most, std::integral_constant<int, 2>());
        else store_rows(std::integral_constant<int, 4>(), std::integral_constant<int, 2>());
    };
    if (!vec) {   // any strides, any alignment, columns that are no multiple of four
#pragma unroll 1
        for (int row = row0; row < end; row += row_step) {
            float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int s = 0; s < splits; s++) {
                float x[4];
                partial(x, (splits == 1 ? from : map_to_cta(from, (uint32_t)s)) + (uint32_t)row * pitch);
#pragma unroll
                for (int j = 0; j < 4; j++) y[j] += x[j];
            }
            if (add1) add_four(y, add1 + row * p.s1[1], p.s1[2], q.add1_vec != 0, valid);
            if (add2) add_four(y, add2 + row * p.s2[1], p.s2[2], q.add2_vec != 0, valid);
            activate(y);
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < valid) out[row * q.so[1] + j * q.so[2]] = (T)y[j];
        }
    } else if (splits == 1) {
        store_all(std::integral_constant<int, 1>());
    } else if (splits == 2) {
        store_all(std::integral_constant<int, 2>());
    } else if (splits <= 4) {
        store_all(std::integral_constant<int, 4>());
    } else {
        store_all(std::integral_constant<int, 8>());
    }
    __syncwarp();
    if (splits > 1) cluster_sync_relaxed();   // nobody leaves while its partial tile may still be read (what was read has been used)
}

struct GemmSlicesLaunch {
    CUtensorMap map_a, map_b;
    GemmSlicesParams p;
    unsigned grid;
    int smem_bytes;
    bool half;
};

struct GemmPersistentLaunch {
    CUtensorMap map_a, map_b, map_c;
    GemmPersistentParams p;
    dim3 grid;
    int smem_bytes;
    bool half;
    bool pair;   // CTA pairs (clusters of two, cta_group::2)
};

// 0 absent, 1 one value per column (row stride 0), 2 a value per element with contiguous rows, 4 one value per
// row (column stride 0), 3 anything else
int classify_addend(const float* ptr, const int64_t* st) {
    if (ptr == nullptr) return 0;
    if (st[1] == 0) return 1;
    if (st[2] == 1) return 2;
    if (st[2] == 0) return 4;
    return 3;
}

}  // namespace

// Column blocks of equal width: n = 320 is two blocks of 160, not 256 + 64 with three quarters of the second empty.
int gemm_persistent_bn(int64_t n) {
    if (const char* e = getenv("KN_GEMM_BN")) {   // (measuring: a fixed block width, a multiple of 32)
        const int v = atoi(e);
        if (v >= 32 && v <= 256 && v % 32 == 0 && n >= v) return v;
    }
    const int64_t blocks = (n + 255) / 256;
    // (several blocks: a multiple of 32, the width of an epilogue chunk, so that no chunk reaches into the
    // next block's columns; a single block is clipped by the store's tensor bounds)
    const int64_t unit = blocks > 1 ? 32 : 16;
    return (int)std::min<int64_t>(((n + blocks - 1) / blocks + unit - 1) / unit * unit, 256);
}

// Tensor maps of the two operands, tiles of 128 rows of A and `b_rows` rows of B, and the parameters that locate a tile
// in them.  False if an operand cannot be read that way.
static bool operand_maps(const GemmParams& g, int b_rows, GemmPersistentParams& p, CUtensorMap* map_a, CUtensorMap* map_b) {
    const bool half = g.half != 0;
    const int64_t align = half ? 8 : 4;            // elements per 16 bytes
    const int block_k = half ? 64 : 32;
    p.a_batch = (g.batch > 1 && g.sa[0] == 0) ? 0 : 1;
    int64_t adims[3] = {g.k, g.m, p.a_batch ? g.batch : 1}, astr[3] = {1, g.sa[1], p.a_batch ? g.sa[0] : align};
    int abox[3] = {block_k, kGpBlockM, 1};
    p.b_batch = (g.batch > 1 && g.sb[0] == 0) ? 0 : 1;
    int64_t bdims[3] = {g.k, g.n, p.b_batch ? g.batch : 1}, bstr[3] = {1, g.sb[2], p.b_batch ? g.sb[0] : align};
    int bbox[3] = {block_k, b_rows, 1};
    // the implicit convolution operand: a 4-D map of the image tensor (channel, x, y, image) whose box is one K
    // block of channels by whole output rows
    int64_t idims[4] = {g.conv_c, g.conv_w, g.conv_h, g.batch}, istr[4] = {1, g.conv_strides[2], g.conv_strides[1], g.conv_strides[0]};
    int ibox[4] = {32, 1, 1, 1};
    if (g.conv_operand != 0) {
        const int rows = g.conv_operand == 1 ? kGpBlockM : b_rows;
        if (half || g.conv_c % 32 != 0 || g.conv_ow < 1 || g.conv_ow > 256 || rows % g.conv_ow != 0 || g.conv_r < 1 || g.conv_s < 1 ||
            g.k != (int64_t)g.conv_r * g.conv_s * g.conv_c)
            return false;
        ibox[1] = g.conv_ow;
        ibox[2] = rows / g.conv_ow;
        p.conv_operand = g.conv_operand;
        p.conv_cblocks = g.conv_c / 32;
        p.conv_s = g.conv_s;
        p.conv_pad_y = g.conv_pad_y;
        p.conv_pad_x = g.conv_pad_x;
        p.conv_ow = g.conv_ow;
    }
    // 4-D operands: the box is one K block by the tile's rows inside one (x, y) entry
    auto operand_4d = [&](const GemmOperand4D& o, const void* base, int rows, int64_t matrix_rows, int32_t* kd_shift, int32_t* rd, int32_t* bi,
                          CUtensorMap* map) {
        if (!o.enabled) return true;
        if (o.kd < 1 || o.rd < 1 || o.bi < 1 || o.strides[0] != 1 || g.conv_operand != 0) return false;
        int shift = 0;
        if (o.kd != g.k) {   // the K offset is split: whole K blocks inside one entry, by a shift
            if (o.kd % block_k != 0 || (o.kd & (o.kd - 1)) != 0) return false;
            while ((1 << shift) < o.kd) shift++;
        }
        // a tile's rows lie inside one entry: an entry's rows are a multiple of the tile's, or the matrix is one entry
        // tall (then rows past its end are past the tensor's extent: zero fill)
        if (o.rd % rows != 0 && o.rd < matrix_rows) return false;
        int box[4] = {block_k, rows, 1, 1};
        *map = half ? tc_make_map_f16(base, 4, o.dims, o.strides, box, true) : tc_make_map(base, 4, o.dims, o.strides, box, true);
        *kd_shift = shift;
        *rd = o.rd;
        *bi = o.bi;
        return true;
    };
    if (!operand_4d(g.a4, g.a, kGpBlockM, g.m, &p.a4_kd_shift, &p.a4_rd, &p.a4_bi, map_a)) return false;
    if (!operand_4d(g.b4, g.b, b_rows, g.n, &p.b4_kd_shift, &p.b4_rd, &p.b4_bi, map_b)) return false;
    if (g.a4.enabled && g.b4.enabled) {
    } else if (g.a4.enabled) {
        *map_b = half ? tc_make_map_f16(g.b, 3, bdims, bstr, bbox, true) : tc_make_map(g.b, 3, bdims, bstr, bbox, true);
    } else if (g.b4.enabled) {
        *map_a = half ? tc_make_map_f16(g.a, 3, adims, astr, abox, true) : tc_make_map(g.a, 3, adims, astr, abox, true);
    } else if (half) {
        *map_a = tc_make_map_f16(g.a, 3, adims, astr, abox, true);
        *map_b = tc_make_map_f16(g.b, 3, bdims, bstr, bbox, true);
    } else {
        *map_a = g.conv_operand == 1 ? tc_make_map(g.a, 4, idims, istr, ibox, true) : tc_make_map(g.a, 3, adims, astr, abox, true);
        *map_b = g.conv_operand == 2 ? tc_make_map(g.b, 4, idims, istr, ibox, true) : tc_make_map(g.b, 3, bdims, bstr, bbox, true);
    }
    return true;
}

std::shared_ptr<void> gemm_persistent_prepare(const GemmParams& g, uint32_t* status_word, int splits, int k_iters_slice,
                                              uint32_t* trace_words) {
    if (g.batch < 1 || g.m < 1 || g.n < 16 || g.k < 1 || splits < 1) return nullptr;
    const bool split = splits > 1;
    const bool half = g.half != 0;
    const int64_t align = half ? 8 : 4;            // elements per 16 bytes
    const int block_k = half ? 64 : 32;
    // dense row-major C whose rows start on 16-byte boundaries (split K: the partial sums [batch][slice][m][n],
    // which the reduction kernel turns into C; addends and activation are applied there)
    if (split) {
        if (g.n % 4 != 0 || ((uintptr_t)g.scratch & 15) != 0 || g.scratch == nullptr) return nullptr;
    } else if (g.sc[2] != 1 || g.sc[1] % align != 0 || (g.batch > 1 && g.sc[0] % align != 0) || ((uintptr_t)g.c & 15) != 0) {
        return nullptr;
    }
    const int m1 = split ? 0 : classify_addend(g.add1, g.s1), m2 = split ? 0 : classify_addend(g.add2, g.s2);
    if (m1 == 3 || m2 == 3) return nullptr;
    auto l = std::make_shared<GemmPersistentLaunch>();
    GemmPersistentParams& p = l->p;
    memset(&p, 0, sizeof(p));
    p.bn = gemm_persistent_bn(g.n);
    p.k_iters = (int)((g.k + block_k - 1) / block_k);
    p.out_half = half && !split ? 1 : 0;
    l->half = half;
    p.n_tiles = (int)((g.n + p.bn - 1) / p.bn);
    // CTA pairs: at least one 256-row tile per pair of SMs, and a reduction long enough
    // for the mainloop to matter (pairs against one CTA a tile, 16384 x 768, 16384 x 3072, 4096 x 4096 and 8192 x 1024 results in f32
    // and f16: 1.13 to 1.25 of the time at 2 and 4 K blocks, where a tile is mostly epilogue and the pair's hand-offs cost more
    // than the operand traffic they save, 0.96 to 1.11 at 12, 0.90 to 1.04 at 16, 0.86 to 0.99 at 20 and 24).
    // KN_GEMM_PAIR=0 in the environment switches pairs off, KN_GEMM_PAIR=1 drops the K condition (A/B measurements).
    // (no K slices; the A operand may be a head split or merge read in place, 42.3 -> 38.5 us on the BERT output
    // projection; with convolution windows as the A operand pairs measured no faster, 127.4 against 126.3 us, and a B
    // operand read in place would need its box halved: those stay on one CTA per tile)
    bool pair = !split && g.conv_operand == 0 && !g.b4.enabled && p.bn % 32 == 0 && p.bn >= 64 && g.m >= 256 &&
                ((g.m + 255) / 256) * p.n_tiles * g.batch >= 74;
    const char* pair_env = getenv("KN_GEMM_PAIR");
    if (pair_env && atoi(pair_env) == 0) pair = false;
    if (!pair_env && p.k_iters < 20) pair = false;
    l->pair = pair;
    p.m_tiles = (int)((g.m + (pair ? 2 : 1) * kGpBlockM - 1) / ((pair ? 2 : 1) * kGpBlockM));
    p.batch = (int)g.batch;
    p.splits = splits;
    p.k_iters_slice = split ? k_iters_slice : p.k_iters;
    if ((int64_t)(splits - 1) * p.k_iters_slice >= p.k_iters) return nullptr;   // an empty slice
    const int64_t total = (int64_t)p.m_tiles * p.n_tiles * g.batch * splits;
    if (total > (1 << 30)) return nullptr;
    p.total_tiles = (int)total;
    p.m = g.m;
    p.n = g.n;
    p.add1 = g.add1;
    p.add2 = g.add2;
    for (int i = 0; i < 3; i++) {
        p.s1[i] = g.s1[i];
        p.s2[i] = g.s2[i];
    }
    p.add1_mode = m1;
    p.add2_mode = m2;
    p.act = split ? 0 : g.act;
    p.status = status_word;
    p.dbg = (volatile uint32_t*)trace_words;
    // KN_GEMM_CLOCKS=1 in the environment: CTA 0 stamps clock64 per tile (MMA thread: tile reached, accumulator free,
    // first K block landed, all MMAs issued; copy-engine thread of the epilogue: accumulator ready, tile stored, cycles
    // spent waiting for staging tiles) and the table of the last launch is printed when the process exits.
    if (getenv("KN_GEMM_CLOCKS")) {
        static long long* table = nullptr;
        if (!table && cudaHostAlloc((void**)&table, (size_t)kGpClockTiles * 64, cudaHostAllocMapped) == cudaSuccess) {
            atexit([] {
                const long long* d = table;
                fprintf(stderr, "gemm_persistent_kernel, CTA 0, SM clock cycles since the MMA thread reached the tile\n"
                                "tile  accumulator_free  first_block_landed  mmas_issued  | accumulator_ready  tile_stored  (staging waits)  | period\n");
                for (int i = 0; i < kGpClockTiles && d[i * 8 + 3]; i++)
                    fprintf(stderr, "%4d  %16lld  %18lld  %11lld  | %17lld  %11lld  %15lld  | %6lld\n", i, d[i * 8 + 1] - d[i * 8], d[i * 8 + 2] - d[i * 8],
                            d[i * 8 + 3] - d[i * 8], d[i * 8 + 4] - d[i * 8], d[i * 8 + 5] - d[i * 8], d[i * 8 + 6], i ? d[i * 8] - d[(i - 1) * 8] : 0);
            });
        }
        if (table) memset(table, 0, (size_t)kGpClockTiles * 64);
        p.clocks = table;
    }
    const int stage_bytes = kGpATileBytes + (pair ? p.bn / 2 : p.bn) * 128;
    // One group where there is nothing to add or compute: stores leave in the order of the columns then, which is what short tiles in
    // f32 are bound by (f16 stores are half as long), and the power that the second group takes is the MMAs'.  One group -> two:
    // 384 x 512 x 512 x 64 87.9 -> 94.7 us (with a staging tile more each 100; one group chosen in the kernel instead of compiled 92), 4096 x
    // 2304 x 64 11.6 -> 13.0, 16384 x 768 x 512 34.0 -> 34.8, x 2048 102.3 -> 102.5.  With a bias 4096 x 2304 x 64 22.0 -> 17.0, x 256 23.9 -> 19.7, x 384
    // 26.1 -> 21.4; f16 16384 x 768 x 128 17.1 -> 15.7, x 640 24.7 -> 23.9.
    p.groups = !pair && !half && g.add1 == nullptr && g.act == 0 ? 1 : 2;
    const int fixed = 1024 + 2 * kGpStageTileBytes + 16 * 8 + 64 + 64;
    p.stages = std::max(2, std::min(6, (227 * 1024 - fixed) / stage_bytes));
    l->smem_bytes = fixed + p.stages * stage_bytes;
    if (!operand_maps(g, pair ? p.bn / 2 : p.bn, p, &l->map_a, &l->map_b)) return nullptr;
    int64_t cdims[3] = {g.n, g.m, g.batch * splits}, cstr[3] = {1, split ? g.n : g.sc[1], split ? g.m * g.n : g.sc[0]};
    int cbox[3] = {32, kGpBlockM, 1};
    if (p.out_half) l->map_c = tc_make_map_f16(g.c, 3, cdims, cstr, cbox, false);
    else l->map_c = tc_make_store_map(split ? g.scratch : g.c, 3, cdims, cstr, cbox);
    l->grid = pair ? dim3(2u * (unsigned)std::min<int64_t>(total, 74), 1, 1) : dim3((unsigned)std::min<int64_t>(total, 148), 1, 1);
    return l;
}

int gemm_persistent_launch(const void* launch, cudaStream_t stream) {
    const GemmPersistentLaunch& l = *(const GemmPersistentLaunch*)launch;
    static std::mutex mu;
    static bool done[64] = {false};
    int device = 0;
    cudaGetDevice(&device);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (device >= 0 && device < 64 && !done[device]) {
            const void* variants[] = {(const void*)gemm_persistent_kernel<false, false, 1>,
                                      (const void*)gemm_persistent_kernel<false, false, 2>, (const void*)gemm_persistent_kernel<true, false, 2>,
                                      (const void*)gemm_persistent_kernel<false, true, 2>, (const void*)gemm_persistent_kernel<true, true, 2>};
            for (const void* v : variants) {
                cudaError_t e = cudaFuncSetAttribute(v, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e != cudaSuccess) return (int)e;
            }
            done[device] = true;
        }
    }
    if (l.pair) {
        // clusters of two CTAs, still with the programmatic edge to the previous kernel
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = l.grid;
        cfg.blockDim = dim3(64u + 128u * (unsigned)l.p.groups);   // (two: see gemm_persistent_prepare)
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
        if (l.half) return (int)cudaLaunchKernelEx(&cfg, gemm_persistent_kernel<true, true, 2>, l.map_a, l.map_b, l.map_c, l.p);
        return (int)cudaLaunchKernelEx(&cfg, gemm_persistent_kernel<false, true, 2>, l.map_a, l.map_b, l.map_c, l.p);
    }
    auto launch_groups = [&](auto kernel) {
        launch_pdl(kernel, dim3(l.grid), dim3(64u + 128u * (unsigned)l.p.groups), (size_t)(l.smem_bytes), stream, l.map_a, l.map_b, l.map_c, l.p);
    };
    if (l.p.groups == 1) launch_groups(gemm_persistent_kernel<false, false, 1>);
    else launch_groups(l.half ? gemm_persistent_kernel<true, false, 2> : gemm_persistent_kernel<false, false, 2>);
    return (int)cudaGetLastError();
}

// Tile width and K slices for gemm_slices_kernel; slices = 0: the matmul is for the persistent kernel.
//
// The line: less than one round of the chip in the persistent kernel's tiles (at most 148 of 128 rows x its block width).
// Within it the cheapest total wins, in SM cycles as clock stamps in the kernel show them: a K block costs its MMAs (bn / 2
// cycles each, four of them) or its bytes at the 65 per cycle that an SM takes from L2, whichever is longer; a CTA 2 500 before
// and 1 300 after its first and last MMAs; the partial tile's way to shared memory 4.5 a column and its way out 25 a column, or,
// with slices, two cluster barriers and the bytes that come from other CTAs, of which an SM takes some 16 per cycle
// (120 x 2304 x 768: 2 slices of 32 columns 8.4 us, 5 of 96 9.0; 640 x 1024 x 2880: 6 slices of 256 columns 16.7 us, 3 of 128
// 18.6).  A round holds fewer CTAs than there are SMs when they come in clusters, which lie inside a GPC (kClusterCtas).
GemmSlices gemm_slices_choose(const GemmParams& g) {
    // CTAs of one per SM that fit the chip at once, by the size of their clusters (cudaOccupancyMaxActiveClusters)
    static const int kClusterCtas[kGsMaxSlices + 1] = {0, 148, 148, 135, 132, 130, 132, 105, 120};
    GemmSlices none{};
    if (g.batch < 1 || g.m < 1 || g.n < 8 || g.k < 1 || g.row_softmax != 0) return none;
    const int64_t m_tiles = (g.m + kGpBlockM - 1) / kGpBlockM;
    const int64_t wide = gemm_persistent_bn(g.n);
    const int64_t persistent_tiles = m_tiles * ((g.n + wide - 1) / wide) * g.batch;
    if (persistent_tiles > 148) return none;
    const int64_t k_blocks = (g.k + (g.half ? 63 : 31)) / (g.half ? 64 : 32);
    GemmSlices best{};
    double best_cost = 0;
    for (int bn = 32; bn <= 256; bn += 32) {
        if (bn > 32 && bn - 32 >= g.n) break;
        if (g.conv_operand == 2 && bn % g.conv_ow != 0) continue;
        if (g.b4.enabled && g.b4.rd % bn != 0 && g.b4.rd < g.n) continue;
        const int64_t tiles = m_tiles * ((g.n + bn - 1) / bn) * g.batch;
        if (tiles > (1 << 24)) continue;
        const double block = std::max({350.0, 2.0 * bn, (kGpATileBytes + 128.0 * bn) / 65.0});
        for (int64_t want = 1; want <= kGsMaxSlices && want <= k_blocks; want++) {
            const int64_t per = (k_blocks + want - 1) / want, slices = (k_blocks + per - 1) / per;
            if (slices != want) continue;
            const double rounds = std::ceil((double)(tiles * slices) / kClusterCtas[slices]);
            const double store = slices > 1 ? 3600.0 + 26.0 * bn * (double)(slices - 1) / (double)slices : 25.0 * bn;
            const double cost = rounds * (3800.0 + per * block + 4.5 * bn + store);
            if (best.slices == 0 || cost < best_cost) {
                best_cost = cost;
                best.slices = (int)slices;
                best.bn = bn;
            }
        }
    }
    return best;
}

std::shared_ptr<void> gemm_slices_prepare(const GemmParams& g, uint32_t* status_word) {
    if (g.slices < 1 || g.slices > kGsMaxSlices || g.slices_bn < 32 || g.slices_bn > 256 || g.slices_bn % 32 != 0) return nullptr;
    if (g.half && (g.add1 != nullptr || g.add2 != nullptr)) return nullptr;
    auto l = std::make_shared<GemmSlicesLaunch>();
    memset(&l->p, 0, sizeof(l->p));
    GemmPersistentParams& p = l->p.g;
    l->half = g.half != 0;
    p.bn = g.slices_bn;
    p.k_iters = (int)((g.k + (l->half ? 63 : 31)) / (l->half ? 64 : 32));
    p.k_iters_slice = (p.k_iters + g.slices - 1) / g.slices;
    p.splits = g.slices;
    if ((int64_t)(p.splits - 1) * p.k_iters_slice >= p.k_iters) return nullptr;   // an empty slice
    p.m_tiles = (int)((g.m + kGpBlockM - 1) / kGpBlockM);
    p.n_tiles = (int)((g.n + p.bn - 1) / p.bn);
    p.batch = (int)g.batch;
    const int64_t ctas = (int64_t)p.m_tiles * p.n_tiles * g.batch * p.splits;
    if (ctas > (1 << 30)) return nullptr;
    p.m = g.m;
    p.n = g.n;
    p.add1 = g.add1;
    p.add2 = g.add2;
    for (int i = 0; i < 3; i++) {
        p.s1[i] = g.s1[i];
        p.s2[i] = g.s2[i];
        l->p.so[i] = g.sc[i];
    }
    p.act = g.act;
    p.status = status_word;
    l->p.out = g.c;
    l->p.a_const = g.a_const;
    l->p.b_const = g.b_const;
    const uintptr_t align = l->half ? 7 : 15;
    auto vec = [&](const void* ptr, const int64_t* st) {
        return ((uintptr_t)ptr & align) == 0 && st[2] == 1 && st[1] % 4 == 0 && st[0] % 4 == 0 ? 1 : 0;
    };
    l->p.out_vec = vec(g.c, g.sc);
    l->p.add1_vec = vec(g.add1, g.s1);
    l->p.add2_vec = vec(g.add2, g.s2);
    l->p.tmem_cols = 32;
    while (l->p.tmem_cols < p.bn) l->p.tmem_cols *= 2;
    const int stage_bytes = kGpATileBytes + p.bn * 128, tile_bytes = kGpBlockM * (p.bn + 4) * 4;
    // (a short slice: no more than half of an SM's shared memory, so that the next kernel's CTA finds room beside it)
    const bool shared_sm = tile_bytes <= 100 * 1024 && (ctas > 148 || p.k_iters_slice * stage_bytes <= 200 * 1024);
    const int room = (shared_sm ? 108 : 224) * 1024;
    p.stages = std::max(1, std::min(std::min(p.k_iters_slice, 8), room / stage_bytes));
    l->smem_bytes = 1024 + std::max(p.stages * stage_bytes, tile_bytes) + 16 * p.stages + 32;
    if (!operand_maps(g, p.bn, p, &l->map_a, &l->map_b)) return nullptr;
    l->grid = (unsigned)ctas;
    return l;
}

int gemm_slices_launch(const void* launch, cudaStream_t stream) {
    const GemmSlicesLaunch& l = *(const GemmSlicesLaunch*)launch;
    static std::mutex mu;
    static bool done[64] = {false};
    int device = 0;
    cudaGetDevice(&device);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (device >= 0 && device < 64 && !done[device]) {
            for (const void* v : {(const void*)gemm_slices_kernel<false>, (const void*)gemm_slices_kernel<true>}) {
                cudaError_t e = cudaFuncSetAttribute(v, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e != cudaSuccess) return (int)e;
            }
            done[device] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(l.grid);
    cfg.blockDim = dim3(kGsThreads);
    cfg.dynamicSmemBytes = (size_t)l.smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)l.p.g.splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = l.p.g.splits > 1 ? 2 : 1;
    if (l.half) return (int)cudaLaunchKernelEx(&cfg, gemm_slices_kernel<true>, l.map_a, l.map_b, l.p);
    return (int)cudaLaunchKernelEx(&cfg, gemm_slices_kernel<false>, l.map_a, l.map_b, l.p);
}

}  // namespace kn
