// Attention over any number of keys for sm_100a: out = softmax(scale * Q . K^T + term) . V without the scores or the
// probabilities ever leaving the SM, one CTA per (batch entry, 128 query rows).  Operands in f32 storage (TF32 on load,
// kind::tf32) or f16 storage (kind::f16); statistics, sums and both accumulators are f32 in either.
//
// The keys are taken 64 at a time.  A block's scores are one of two accumulators of 64 columns in tensor memory; its
// probabilities take the place of the scores (f16: packed, half the columns) and are the A operand of the second MMA, whose
// accumulator of up to 128 columns is kept over all blocks.  Exponentials are taken against a reference that follows the
// row's running maximum only when that has risen by more than 8 (in powers of two): then the row's accumulator and sum are
// rescaled (once the block before has been added), which after the first few blocks hardly ever happens; the quotient does
// not depend on the reference.
//
//   warps 0..3      softmax: a row per thread, all 64 columns of it, so nothing is exchanged (few blocks on few CTAs: eight warps, PAIRED)
//   warp 4, a lane  producer: Q once, keys and values of a block through two buffers each (one where two do not fit)
//   warp 5, a lane  MMA issuer: the next block's score MMAs go ahead of this block's context MMAs, under its exponentials
//
// Two CTAs share an SM: 256 columns of tensor memory, some 100 KB of shared memory (head dimensions up to 64 in f32 or 128 in
// f16; larger ones run one CTA per SM), 192 threads with 160 registers: a row's 64 scores stay in them.  (With blocks of 128
// keys, one accumulator, and a row on two warps the phases of a block followed one another: 6 000 cycles of a CTA for 128 keys,
// 5 000 now, 240 to 280 bytes of registers spilled, a barrier of all warps for every maximum.)
//
// Measured (kernel_bench's attention_causal_f16, attention_latent and attention_short_f16), one accumulator of 128 keys -> now:
// 32 heads of 2048 causal rows, f16, d = 128: 94 -> 69 us, 10 of them flash_finite_kernel; 8 heads of 4096 rows, f32, d = 40:
// 119 -> 74 us; 32 heads of 333 causal rows, f16, d = 128: 19.5 -> 16.4 us.
// What bounds it: f32, the context MMAs (80 cycles for 8 keys with A from tensor memory, whatever the number of columns: 1 300 of
// the 2 500 cycles that an SM takes for 128 keys) next to the exponentials (1 024 at 16 a cycle).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>

#include "../tc.h"
#include "tc_host.h"
#include "tc_ptx.cuh"
#include "launch.cuh"

namespace kn {

namespace {

using namespace tcp;

constexpr int kFlRows = 128, kFlKeys = 64;
constexpr int kFlTableKeys = 128;          // keys of a block in the planner's table of a constant term
constexpr int kFlQBytes = kFlRows * 128, kFlKeyBytes = kFlKeys * 128;   // a panel: rows of 128 bytes
constexpr int kFlTmemCols = 256, kFlOutCol = 128;
constexpr int kFlExchangeBytes = 2 * 2 * kFlRows * 4;   // (PAIRED)
constexpr float kLog2e = 1.44269504088896340736f;
constexpr float kRiseLimit = 8.0f;
constexpr float kHalfSumBelow = -1024.f;   // f16 values are one apart here
constexpr uint32_t kFlSleepNs = 1000;

struct FlashParams {
    int32_t m, n, batch, m_tiles, key_blocks, table_blocks;
    int32_t key_slots, value_slots;  // buffers of a block's keys, of its values: one or two
    int32_t qk_blocks, qk_steps;     // 128-byte blocks of a row of Q; instructions of 32 bytes along it
    int32_t dv, v_panels, out_cols;  // columns of V, 128-byte panels of them, N of the context MMAs
    int32_t a_bi, b_bi, v_bi;        // batch entry bt -> map coordinates (bt % bi, bt / bi)
    float scale;
    void* out;
    int32_t out_heads;               // out[bt / out_heads][bt % out_heads][row][column] with strides out_s (the last 1)
    int64_t out_s[3];
    const void* term;                // additive term [batch][m][n], or null
    int64_t term_s[3];
    int32_t term_cols;               // columns of a row that may be read: n, or more with padding
    // of a constant term that all batch entries share: per row block the number of key blocks to visit (what follows is
    // -infinity), then per key block what the term is there: 0 zero, 2 -infinity, 1 anything else (it is read); else null
    const int16_t* term_blocks;
    const int32_t* not_finite;       // [batch][key blocks] of flash_finite_kernel, or null: no block is left out
    uint32_t* status;
};

__device__ __forceinline__ void mma_f16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void arrive_one(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_loads_done() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_stores_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// PAIRED: eight softmax warps, of which four take the even blocks and four the odd ones; of a pair of blocks they exchange the rows'
// maxima, so that both go by one reference.  For grids that leave an SM one CTA, whose blocks would follow one another.
template <bool HALF, bool TERM, bool PAIRED>
__global__ void __launch_bounds__(PAIRED ? 320 : 192, PAIRED ? 1 : 2)
flash_attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ FlashParams p) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int kElems = HALF ? 64 : 32;   // elements per 128 bytes
    constexpr int kSoftmaxWarps = PAIRED ? 8 : 4;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t k_bytes = (uint32_t)(p.qk_blocks * kFlKeyBytes), v_bytes = (uint32_t)(p.v_panels * kFlKeyBytes);
    const uint32_t k_base = base + (uint32_t)(p.qk_blocks * kFlQBytes);
    const uint32_t v_base = k_base + (uint32_t)p.key_slots * k_bytes;
    const uint32_t bars = v_base + (uint32_t)p.value_slots * v_bytes;
    // (of two: one per parity of the block)
    const uint32_t q_full = bars, pv_done = bars + 8u, k_full = bars + 24u, v_full = bars + 40u, s_full = bars + 56u, p_ready = bars + 72u, slot_addr = bars + 88u;
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + (slot_addr - base));
    volatile int* abandon = (volatile int*)(gen_base + (slot_addr + 4u - base));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (uint32_t b = 0; b < 16u; b += 8u) {
            mbar_init(pv_done + b, 1);
            mbar_init(k_full + b, 1);
            mbar_init(v_full + b, 1);
            mbar_init(s_full + b, 1);
            mbar_init(p_ready + b, kSoftmaxWarps);
        }
        *abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kSoftmaxWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"((uint32_t)kFlTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_s = *tmem_slot, tmem_o = tmem_s + (uint32_t)kFlOutCol;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // the last row blocks first: under a causal mask they have the most keys
    const int bt = (int)(blockIdx.x % (unsigned)p.batch), mt = p.m_tiles - 1 - (int)(blockIdx.x / (unsigned)p.batch);
    const int16_t* blocks_of = TERM && p.term_blocks ? p.term_blocks + (int64_t)mt * (p.table_blocks + 1) : nullptr;   // (a constant)
    constexpr int kTableStep = kFlTableKeys / kFlKeys;
    int n_table = blocks_of ? (int)blocks_of[0] : p.table_blocks;
    auto block_cols = [&](int j) { return min(kFlKeys, (p.n - j * kFlKeys + 31) & ~31); };   // (past n: zero fill, masked below)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (TERM && p.not_finite && n_table < p.table_blocks) {   // up to the last masked block that does not give exact zeros
        const int32_t* flags = p.not_finite + (int64_t)bt * p.table_blocks;
        int last = 0;
        for (int j = n_table + lane; j < p.table_blocks; j += 32) last = flags[j] != 0 ? j + 1 : last;
        n_table = max(n_table, __reduce_max_sync(0xffffffffu, last));
    }
    const int n_blocks = min(n_table * kTableStep, p.key_blocks);

    if (warp == kSoftmaxWarps) {
        if (elect_one()) {
            // ---------------- producer
            const uint32_t q_bytes = (uint32_t)(p.qk_blocks * kFlQBytes);
            mbar_expect_tx(q_full, q_bytes);
            for (int b = 0; b < p.qk_blocks; b++)
                tma_load_4d(base + (uint32_t)(b * kFlQBytes), &map_q, q_full, b * kElems, mt * kFlRows, bt % p.a_bi, bt / p.a_bi);
            const int k2 = bt % p.b_bi, k3 = bt / p.b_bi, v2 = bt % p.v_bi, v3 = bt / p.v_bi;
            auto keys = [&](int j) -> bool {
                const int used = j - p.key_slots;   // the block whose keys lay there: its scores are complete
                if (used >= 0 && !mbar_wait(s_full + 8u * (used & 1), (uint32_t)((used >> 1) & 1), abandon, p.status, 51, kWaitCycles, kFlSleepNs)) return false;
                const uint32_t to = k_base + (p.key_slots == 2 ? (uint32_t)(j & 1) * k_bytes : 0u);
                mbar_expect_tx(k_full + 8u * (j & 1), k_bytes);
                for (int b = 0; b < p.qk_blocks; b++)
                    tma_load_4d(to + (uint32_t)(b * kFlKeyBytes), &map_k, k_full + 8u * (j & 1), b * kElems, j * kFlKeys, k2, k3);
                return true;
            };
            bool ok = keys(0);
            for (int j = 0; j < n_blocks && ok; j++) {
                if (j + 1 < n_blocks && !keys(j + 1)) break;
                const int used = j - p.value_slots;
                if (used >= 0 && !mbar_wait(pv_done + 8u * (used & 1), (uint32_t)((used >> 1) & 1), abandon, p.status, 52, kWaitCycles, kFlSleepNs)) break;
                const uint32_t to = v_base + (p.value_slots == 2 ? (uint32_t)(j & 1) * v_bytes : 0u);
                mbar_expect_tx(v_full + 8u * (j & 1), v_bytes);
                for (int b = 0; b < p.v_panels; b++)
                    tma_load_4d(to + (uint32_t)(b * kFlKeyBytes), &map_v, v_full + 8u * (j & 1), b * kElems, j * kFlKeys, v2, v3);
            }
        }
    } else if (warp == kSoftmaxWarps + 1) {
        if (elect_one()) {
            // ---------------- MMA issuer: f32 accumulate, M = 128; Q and the keys K-major, V with its columns contiguous
            // (bit 16: the MN-major B operand)
            const uint32_t fmt = HALF ? 0u : 2u;
            const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(kFlRows >> 4) << 24);
            const uint32_t idesc_o = idesc | (1u << 16) | ((uint32_t)(p.out_cols >> 3) << 17);
            // MN-major B: panels of 128 bytes of columns lie `leading byte offset` apart, groups of keys `stride byte
            // offset`: eight keys and the 128-byte swizzle for 16-bit elements, four and the swizzle in 32-byte pieces for
            // 32-bit ones (see attention.cu)
            const uint64_t v_desc = ((uint64_t)(kFlKeyBytes >> 4) << 16) | ((uint64_t)((HALF ? 1024 : 512) >> 4) << 32) | ((uint64_t)1 << 46) |
                                    ((uint64_t)(HALF ? 2 : 1) << 61);
            constexpr int kStepKeys = HALF ? 16 : 8, kStepCols = 8;   // keys of an instruction; their columns in tensor memory
            auto scores = [&](int j) -> bool {
                const uint32_t b = (uint32_t)(j & 1);
                if (!mbar_wait(k_full + 8u * b, (uint32_t)((j >> 1) & 1), abandon, p.status, 54, kWaitCycles, kFlSleepNs)) return false;
                // (the probabilities of the block before the last lie where the scores go)
                if (j > 1 && !mbar_wait(pv_done + 8u * b, (uint32_t)(((j - 2) >> 1) & 1), abandon, p.status, 55, kWaitCycles, kFlSleepNs)) return false;
                tc_fence_after();
                const uint32_t idesc_s = idesc | ((uint32_t)(block_cols(j) >> 3) << 17);
                const uint32_t from = k_base + (p.key_slots == 2 ? b * k_bytes : 0u);
                for (int s = 0; s < p.qk_steps; s++) {
                    const uint64_t da = smem_desc_sw128(base + (uint32_t)((s >> 2) * kFlQBytes)) + 2u * (s & 3);
                    const uint64_t db = smem_desc_sw128(from + (uint32_t)((s >> 2) * kFlKeyBytes)) + 2u * (s & 3);
                    if (HALF) mma_f16(tmem_s + b * kFlKeys, da, db, idesc_s, s != 0 ? 1u : 0u);
                    else mma_tf32(tmem_s + b * kFlKeys, da, db, idesc_s, s != 0 ? 1u : 0u);
                }
                mma_commit(s_full + 8u * b);
                return true;
            };
            bool ok = mbar_wait(q_full, 0, abandon, p.status, 53, kWaitCycles, kFlSleepNs) && scores(0);
            for (int j = 0; j < n_blocks && ok; j++) {
                const uint32_t b = (uint32_t)(j & 1), parity = (uint32_t)((j >> 1) & 1);
                if (j + 1 < n_blocks && !scores(j + 1)) break;   // under this block's exponentials
                if (!mbar_wait(v_full + 8u * b, parity, abandon, p.status, 56, kWaitCycles, kFlSleepNs)) break;
                if (!mbar_wait(p_ready + 8u * b, parity, abandon, p.status, 57, kWaitCycles, kFlSleepNs)) break;
                tc_fence_after();
                const uint32_t from = v_base + (p.value_slots == 2 ? b * v_bytes : 0u);
                const int cols = block_cols(j);
                for (int s = 0; s < cols / kStepKeys; s++) {
                    const uint64_t db = v_desc | (uint64_t)(((from + (uint32_t)(s * kStepKeys * 128)) & 0x3FFFFu) >> 4);
                    if (HALF) mma_f16_a_tmem(tmem_o, tmem_s + b * kFlKeys + (uint32_t)(s * kStepCols), db, idesc_o, (j | s) != 0 ? 1u : 0u);
                    else mma_tf32_a_tmem(tmem_o, tmem_s + b * kFlKeys + (uint32_t)(s * kStepCols), db, idesc_o, (j | s) != 0 ? 1u : 0u);
                }
                mma_commit(pv_done + 8u * b);
            }
        }
    } else {
        // ---------------- softmax
        const int quarter = PAIRED ? warp & 3 : warp, group = warp >> 2, row_in_tile = quarter * 32 + lane, row = mt * kFlRows + row_in_tile;
        float* exchange = (float*)(gen_base + (bars + 128u - base));   // [2][group][row]
        const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
        const uint32_t my_o = tmem_o + lane_bits;
        using T = typename std::conditional<HALF, __half, float>::type;
        const T* term_row = TERM ? (const T*)p.term + bt * p.term_s[0] + (int64_t)min(row, p.m - 1) * p.term_s[1] : nullptr;
        auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) -> bool {   // one lane polls
            uint32_t good = 1;
            if (lane == 0) good = mbar_wait(bar, parity, abandon, p.status, code, kWaitCycles, kFlSleepNs) ? 1u : 0u;
            good = __shfl_sync(0xffffffffu, good, 0);
            tc_fence_after();
            return good != 0;
        };
        // one value a row against the other group's, if everybody goes on; `turn` alternates from call to call
        auto meet = [&](bool good, int turn, float& mine_, float& others) -> bool {
            exchange[((turn & 1) * 2 + group) * kFlRows + row_in_tile] = mine_;
            uint32_t all;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t"
                "setp.ne.u32 p, %1, 0;\n\t"
                "bar.red.and.pred q, 1, 256, p;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(all)
                : "r"((uint32_t)good)
                : "memory");
            others = exchange[((turn & 1) * 2 + (group ^ 1)) * kFlRows + row_in_tile];
            return all != 0;
        };
        // x in units of its exponent: with a term  x = scale * s + term, exponent (x - ref) * log2(e); without one x = s
        const float unit = TERM ? kLog2e : p.scale * kLog2e;
        float seen = -INFINITY, ref = 0.f, sum = 0.f;
        bool ok = true, far = false;   // far: a row of the warp has a reference of the lowest values' size
        constexpr int kStep = PAIRED ? 2 : 1;
        for (int first_j = 0; first_j < n_blocks; first_j += kStep) {
            const int j = first_j + (PAIRED ? group : 0);
            const bool mine = !PAIRED || j < n_blocks;
            const uint32_t b = (uint32_t)(j & 1);
            const uint32_t my_s = tmem_s + lane_bits + b * kFlKeys;
            bool good = true;
            if constexpr (PAIRED) {   // (nobody leaves alone: see `meet`)
                good = ok && (!mine || wait(s_full + 8u * b, (uint32_t)((j >> 1) & 1), 58));
            } else {
                if (!wait(s_full + 8u * b, (uint32_t)((j >> 1) & 1), 58)) { ok = false; break; }
            }
            uint32_t v[2][32];
            float top = -INFINITY;
            bool plain = false;   // a block whose term is zero throughout: scores as without a term
            if (!PAIRED || (mine && good)) {
                tmem_load_32_nowait(my_s, v[0]);
                tmem_load_32_nowait(my_s + 32u, v[1]);
                tmem_loads_done();
                const int col0 = j * kFlKeys;
                if (TERM) {
                    const int kind = blocks_of == nullptr ? 1 : (int)blocks_of[1 + j / kTableStep];
                    if (kind == 0 && p.scale > 0.f) {
                        plain = true;
                    } else if (kind != 1) {
                        const float same = kind == 2 ? -INFINITY : 0.f;
#pragma unroll
                        for (int i = 0; i < 64; i++) v[i >> 5][i & 31] = __float_as_uint(fmaf(p.scale, __uint_as_float(v[i >> 5][i & 31]), same));
                    } else {
                        const T* t = term_row + (int64_t)col0 * p.term_s[2];
                        const bool vec = p.term_s[2] == 1 && col0 + 64 <= p.term_cols && ((uintptr_t)t & 15) == 0;
#pragma unroll
                        for (int c = 0; c < 2; c++) {
#pragma unroll
                            for (int i = 0; i < 32; i += 8) {
                                float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                                if (vec) {
                                    if (HALF) {
                                        const uint4 u = __ldg((const uint4*)(t + c * 32 + i));
                                        const __half2* h = (const __half2*)&u;
#pragma unroll
                                        for (int q = 0; q < 4; q++) {
                                            const float2 f = __half22float2(h[q]);
                                            a[2 * q] = f.x, a[2 * q + 1] = f.y;
                                        }
                                    } else {
#pragma unroll
                                        for (int q = 0; q < 2; q++) {
                                            const float4 f = __ldg((const float4*)(t + c * 32 + i) + q);
                                            a[4 * q] = f.x, a[4 * q + 1] = f.y, a[4 * q + 2] = f.z, a[4 * q + 3] = f.w;
                                        }
                                    }
                                } else {
#pragma unroll
                                    for (int q = 0; q < 8; q++)
                                        if (col0 + c * 32 + i + q < p.n) a[q] = (float)t[(int64_t)(c * 32 + i + q) * p.term_s[2]];
                                }
#pragma unroll
                                for (int q = 0; q < 8; q++) {
                                    float x = fmaf(p.scale, __uint_as_float(v[c][i + q]), a[q]);
                                    // Far below anything a row with an unmasked key looks at, f16 sums are rounded as such: a row
                                    // that is masked by f16's lowest value throughout has the same sum, or -infinity, everywhere.
                                    if (HALF && x < kHalfSumBelow) x = __half2float(__float2half_rn(x));
                                    v[c][i + q] = __float_as_uint(x);
                                }
                            }
                        }
                    }
                }
                if (col0 + 64 > p.n) {   // columns past the last key
#pragma unroll
                    for (int i = 0; i < 64; i++)
                        if (col0 + i >= p.n) v[i >> 5][i & 31] = 0xFF800000u;
                }
#pragma unroll
                for (int i = 0; i < 64; i++) top = fmaxf(top, __uint_as_float(v[i >> 5][i & 31]));
                if (plain) top *= p.scale;
            }
            if (PAIRED) {
                float other;
                ok = meet(good, first_j >> 1, top, other);
                if (!ok) break;
                top = fmaxf(top, other);
            }
            // a row whose scores were all -infinity so far has no reference yet (and zeros in its sum and output)
            const bool first = seen == -INFINITY;
            seen = fmaxf(seen, top);
            const bool rise = first || (top - ref) * unit > kRiseLimit;
            if (__any_sync(0xffffffffu, rise)) {
                const float next = rise && seen > -INFINITY ? seen : ref;
                const float factor = rise && !first ? exp2_approx((ref - next) * unit) : 1.f;
                ref = next;
                if (TERM) far = __any_sync(0xffffffffu, !(fabsf(ref) < 1e30f));
                sum *= factor;
                if (first_j > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
                    const int before = first_j - 1;   // (is still being added)
                    int chunks = (p.out_cols + 31) >> 5;
                    if constexpr (PAIRED) {
                        ok = wait(pv_done + 8u * (before & 1), (uint32_t)((before >> 1) & 1), 59);
                        chunks = ok ? chunks : 0;
                    } else {
                        if (!wait(pv_done + 8u * (b ^ 1u), (uint32_t)((before >> 1) & 1), 59)) { ok = false; break; }
                    }
                    for (int c = PAIRED ? group : 0; c < chunks; c += kStep) {
                        uint32_t o[32];
                        tmem_load_32(my_o + (uint32_t)(c * 32), o);
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                        tmem_store_32(my_o + (uint32_t)(c * 32), o);
                    }
                }
            }
            if (PAIRED) {   // (a group's half of the output is rescaled before the other's block is added)
                tmem_stores_done();
                tc_fence_before();
                __syncwarp();
                if (ok && lane == 0 && first_j + (group ^ 1) < n_blocks) arrive_one(p_ready + 8u * (b ^ 1u));
                if (!ok || !mine) continue;
            }
            auto exponentials = [&](auto exponent) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float e0 = exp2_approx(exponent(__uint_as_float(v[c][i]))), e1 = exp2_approx(exponent(__uint_as_float(v[c][i + 1])));
                        if (HALF) {
                            sum += e0 + e1;
                            const __half2 h = __floats2half2_rn(e0, e1);
                            v[0][c * 16 + (i >> 1)] = *(const uint32_t*)&h;
                        } else {
                            // rounded to the operand's eleven bits here, so that the sum is of what the MMAs see
                            uint32_t r0, r1;
                            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r0) : "f"(e0));
                            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r1) : "f"(e1));
                            sum += __uint_as_float(r0) + __uint_as_float(r1);
                            v[c][i] = r0, v[c][i + 1] = r1;
                        }
                    }
                }
            };
            if (TERM && plain && far) {
                // (a row masked by the lowest value so far: its reference times log2(e) would overflow)
#pragma unroll
                for (int i = 0; i < 64; i++) v[i >> 5][i & 31] = __float_as_uint(p.scale * __uint_as_float(v[i >> 5][i & 31]));
                plain = false;
            }
            const float shift = -ref * unit, factor = plain ? p.scale * unit : unit;
            if (TERM && !plain) exponentials([&](float x) { return (x - ref) * unit; });   // (the lowest finite value times log2(e) would overflow)
            else exponentials([&](float x) { return fmaf(x, factor, shift); });
            if (HALF) {
                tmem_store_32(my_s, v[0]);
            } else {
                tmem_store_32(my_s, v[0]);
                tmem_store_32(my_s + 32u, v[1]);
            }
            tmem_stores_done();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_one(p_ready + 8u * b);
        }
        ok = ok && wait(pv_done + 8u * ((n_blocks - 1) & 1), (uint32_t)(((n_blocks - 1) >> 1) & 1), 59);
        if (PAIRED) {
            float other;
            ok = meet(ok, (n_blocks + 1) >> 1, sum, other);
            sum = group == 0 ? sum + other : other + sum;
        }
        if (ok) {
            const float inv = 1.f / sum;
            T* dst = (T*)p.out + (bt / p.out_heads) * p.out_s[0] + (bt % p.out_heads) * p.out_s[1] + (int64_t)row * p.out_s[2];
            for (int c = PAIRED ? group : 0; c < (p.dv + 31) >> 5; c += kStep) {
                uint32_t o[32];
                tmem_load_32(my_o + (uint32_t)(c * 32), o);
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    if (row >= p.m || c * 32 + i >= p.dv) continue;
                    float f[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) f[q] = __uint_as_float(o[i + q]) * inv;
                    if (HALF) {
                        uint32_t h[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const __half2 pair = __floats2half2_rn(f[2 * q], f[2 * q + 1]);
                            h[q] = *(const uint32_t*)&pair;
                        }
                        *(uint4*)(dst + c * 32 + i) = make_uint4(h[0], h[1], h[2], h[3]);
                    } else {
                        *(float4*)(dst + c * 32 + i) = make_float4(f[0], f[1], f[2], f[3]);
                        *(float4*)(dst + c * 32 + i + 4) = make_float4(f[4], f[5], f[6], f[7]);
                    }
                }
                __syncwarp();
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == kSoftmaxWarps) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"((uint32_t)kFlTmemCols) : "memory");
    }
}

// Per key block of 128: does a key or a value of it hold a NaN or an infinity?  A block that the term masks throughout may
// be left out only if not: -infinity added to a score of NaN or infinity, and a probability of 0 times a value of either,
// are NaN.  One pass over K and V: 10 us for 32 heads of 2048 x 128 in f16.
struct FiniteParams {
    const void* base[2];   // keys, values: row r of entry bt at (bt % bi) * s_x + (bt / bi) * s_y + r * s_row
    int64_t s_row[2], s_x[2], s_y[2];
    int32_t bi[2], cols[2];
    int32_t n, key_blocks;
    int32_t* flags;
};

template <bool HALF>
__global__ void __launch_bounds__(256) flash_finite_kernel(const __grid_constant__ FiniteParams p) {
    pdl_enter();
    constexpr int kSize = HALF ? 2 : 4;
    const int j = (int)(blockIdx.x % (unsigned)p.key_blocks), bt = (int)(blockIdx.x / (unsigned)p.key_blocks);
    const int rows = min(kFlTableKeys, p.n - j * kFlTableKeys);
    auto exponent_full = [](uint32_t w) {
        return HALF ? (w & 0x7C00u) == 0x7C00u || (w & 0x7C000000u) == 0x7C000000u : (w & 0x7F800000u) == 0x7F800000u;
    };
    bool found = false;
#pragma unroll
    for (int o = 0; o < 2; o++) {
        const char* base = (const char*)p.base[o] + ((bt % p.bi[o]) * p.s_x[o] + (bt / p.bi[o]) * p.s_y[o] + (int64_t)j * kFlTableKeys * p.s_row[o]) * kSize;
        const int chunks = p.cols[o] * kSize / 16, row_step = 256 / chunks, chunk_step = 256 % chunks;
        int r = threadIdx.x / chunks, c = threadIdx.x % chunks;
#pragma unroll 8
        for (int i = threadIdx.x; i < rows * chunks; i += 256) {
            const uint4 u = *(const uint4*)(base + r * p.s_row[o] * kSize + c * 16);
            found = found | exponent_full(u.x) | exponent_full(u.y) | exponent_full(u.z) | exponent_full(u.w);
            r += row_step, c += chunk_step;
            if (c >= chunks) c -= chunks, r++;
        }
    }
    const int any = __syncthreads_or(found ? 1 : 0);
    if (threadIdx.x == 0) p.flags[blockIdx.x] = any;
}

struct FlashLaunch {
    CUtensorMap map_q, map_k, map_v;
    FlashParams p;
    FiniteParams finite;
    unsigned grid;
    int smem_bytes;
    bool half, paired;
};

// Shared memory with `key_slots` and `value_slots` buffers
int flash_smem_bytes(int64_t k, int64_t dv, bool half, int key_slots, int value_slots) {
    const int64_t elems = half ? 64 : 32, k_panels = (k + elems - 1) / elems, v_panels = (dv + elems - 1) / elems;
    return (int)(1024 + k_panels * kFlQBytes + (key_slots * k_panels + value_slots * v_panels) * kFlKeyBytes + 128);
}

}  // namespace

bool flash_attention_fits(int64_t batch, int64_t m, int64_t n, int64_t k, int64_t dv, bool half) {
    if (batch < 1 || m < 1 || n < 1 || k < 8 || dv < 8) return false;
    if (k > 128 || dv > 128 || k % 8 != 0 || dv % 8 != 0 || n > (1 << 21) || m > (1 << 24)) return false;
    return batch * ((m + kFlRows - 1) / kFlRows) < (1ll << 30) && flash_smem_bytes(k, dv, half, 1, 1) <= 227 * 1024;
}

std::shared_ptr<void> flash_attention_prepare(const GemmParams& g, uint32_t* status_word) {
    const bool half = g.half != 0;
    const int64_t align = half ? 8 : 4, elems = half ? 64 : 32;
    if (g.conv_operand != 0 || g.splits > 1 || g.add2 || g.act != 0 || g.row_softmax != 3 || !g.values || !g.values_mn) return nullptr;
    if (!flash_attention_fits(g.batch, g.m, g.n, g.k, g.values_cols, half)) return nullptr;
    if (g.out_heads < 1 || g.sc[0] % align != 0 || g.sc[1] % align != 0 || g.sc[2] % align != 0 || ((uintptr_t)g.c & 15) != 0) return nullptr;
    auto l = std::make_shared<FlashLaunch>();
    FlashParams& p = l->p;
    memset(&p, 0, sizeof(p));
    l->half = half;
    p.m = (int)g.m;
    p.n = (int)g.n;
    p.batch = (int)g.batch;
    p.m_tiles = (int)((g.m + kFlRows - 1) / kFlRows);
    p.key_blocks = (int)((g.n + kFlKeys - 1) / kFlKeys);
    p.table_blocks = (int)((g.n + kFlTableKeys - 1) / kFlTableKeys);
    p.qk_blocks = (int)((g.k + elems - 1) / elems);
    p.qk_steps = (int)((g.k + elems / 4 - 1) / (elems / 4));
    p.dv = (int)g.values_cols;
    p.v_panels = (int)((g.values_cols + elems - 1) / elems);
    p.out_cols = (p.dv + 15) / 16 * 16;
    p.scale = g.softmax_scale;
    p.out = g.c;
    p.out_heads = g.out_heads;
    for (int i = 0; i < 3; i++) p.out_s[i] = g.sc[i];
    p.term = g.add1;
    for (int i = 0; i < 3; i++) p.term_s[i] = g.s1[i];
    p.term_cols = g.term_cols;
    p.term_blocks = (const int16_t*)g.term_blocks;
    p.not_finite = (const int32_t*)g.scratch;
    p.status = status_word;
    FiniteParams& f = l->finite;
    memset(&f, 0, sizeof(f));
    f.n = p.n;
    f.key_blocks = p.table_blocks;
    f.flags = (int32_t*)g.scratch;
    // an operand [batch, rows, k] as a 4-D map (K offset, row, x, y): a head split read in place as it is, a plain one with
    // x = the batch entry (bi = batch + 1: coordinates (bt, 0))
    auto operand = [&](const GemmOperand4D& o, const void* base, int box_rows, int64_t rows, int64_t cols, int64_t s_batch, int64_t s_row, int64_t s_col,
                       bool mn_major, CUtensorMap* map, int32_t* bi, int scanned) {
        int box[4] = {(int)elems, box_rows, 1, 1};
        int64_t dims[4] = {cols, rows, g.batch, 1}, strides[4] = {1, s_row, s_batch, align};
        if (o.enabled) {
            if (o.kd != cols || o.rd < rows || o.strides[0] != 1) return false;
            for (int i = 0; i < 4; i++) dims[i] = o.dims[i], strides[i] = o.strides[i];
            *bi = o.bi;
        } else {
            if (s_col != 1 || (rows > 1 && (s_row <= 0 || s_row % align != 0)) || (g.batch > 1 && (s_batch <= 0 || s_batch % align != 0))) return false;
            *bi = (int)g.batch + 1;
        }
        if (((uintptr_t)base & 15) != 0) return false;
        if (scanned >= 0) {
            f.base[scanned] = base;
            f.s_row[scanned] = strides[1], f.s_x[scanned] = strides[2], f.s_y[scanned] = strides[3];
            f.bi[scanned] = *bi;
            f.cols[scanned] = (int32_t)cols;
        }
        if (half) *map = tc_make_map_f16(base, 4, dims, strides, box, true);
        else if (mn_major) *map = tc_make_map_mn_major(base, 4, dims, strides, box);
        else *map = tc_make_map(base, 4, dims, strides, box, true);
        return true;
    };
    if (!operand(g.a4, g.a, kFlRows, g.m, g.k, g.sa[0], g.sa[1], g.sa[2], false, &l->map_q, &p.a_bi, -1)) return nullptr;
    if (!operand(g.b4, g.b, kFlKeys, g.n, g.k, g.sb[0], g.sb[2], g.sb[1], false, &l->map_k, &p.b_bi, 0)) return nullptr;
    if (!operand(g.v4, g.values, kFlKeys, g.n, g.values_cols, g.values_strides[0], g.values_strides[1], g.values_strides[2], true, &l->map_v, &p.v_bi, 1))
        return nullptr;
    l->grid = (unsigned)(g.batch * p.m_tiles);
    // Two to four blocks with a term where an SM has one CTA.  One group of softmax warps -> two, causal f16: 32 heads of 128 rows, d = 64 9.4 -> 7.9 us, d =
    // 128 10.6 -> 8.9; 256 rows 11.6 -> 10.6 and 13.2 -> 11.7.  With more blocks the next block's scores under this block's exponentials gain
    // more (8 heads of 512 rows 14.3 -> 15.7, f32 8 of 1024 rows 18.4 -> 24.2), and without a term the exponentials are short: 2 of 1590 rows,
    // 157 keys 6.2 -> 7.2.
    l->paired = p.term != nullptr && l->grid <= 148 && p.key_blocks > 1 && p.key_blocks <= 4 && flash_smem_bytes(g.k, g.values_cols, half, 1, 1) + kFlExchangeBytes <= 227 * 1024;
    // two buffers of each where two CTAs of it share an SM (or none would with one)
    const int half_sm = 113 * 1024, whole_sm = 227 * 1024 - (l->paired ? kFlExchangeBytes : 0);
    p.key_slots = p.value_slots = 1;
    const int limit = !l->paired && flash_smem_bytes(g.k, g.values_cols, half, 1, 1) <= half_sm ? half_sm : whole_sm;
    if (flash_smem_bytes(g.k, g.values_cols, half, 1, 2) <= limit) p.value_slots = 2;
    if (flash_smem_bytes(g.k, g.values_cols, half, 2, p.value_slots) <= limit) p.key_slots = 2;
    l->smem_bytes = flash_smem_bytes(g.k, g.values_cols, half, p.key_slots, p.value_slots) + (l->paired ? kFlExchangeBytes : 0);
    return l;
}

using FlashKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, FlashParams);
template <bool PAIRED>
static FlashKernel flash_kernel(bool half, bool term) {
    return half ? (term ? flash_attention_kernel<true, true, PAIRED> : flash_attention_kernel<true, false, PAIRED>)
                : (term ? flash_attention_kernel<false, true, PAIRED> : flash_attention_kernel<false, false, PAIRED>);
}

int flash_attention_launch(const void* launch, cudaStream_t stream) {
    auto kernel = [](bool half, bool term, bool paired) { return paired ? flash_kernel<true>(half, term) : flash_kernel<false>(half, term); };
    const FlashLaunch& l = *(const FlashLaunch*)launch;
    static std::mutex mu;
    static bool done[64] = {false};
    int device = 0;
    cudaGetDevice(&device);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (device >= 0 && device < 64 && !done[device]) {
            for (FlashKernel v : {kernel(false, false, false), kernel(false, true, false), kernel(true, false, false), kernel(true, true, false),
                                  kernel(false, false, true), kernel(false, true, true), kernel(true, false, true), kernel(true, true, true)}) {
                cudaError_t e = cudaFuncSetAttribute(v, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e != cudaSuccess) return (int)e;
            }
            done[device] = true;
        }
    }
    if (l.finite.flags) {
        const dim3 blocks((unsigned)l.p.batch * (unsigned)l.p.table_blocks);
        launch_pdl(l.half ? flash_finite_kernel<true> : flash_finite_kernel<false>, blocks, dim3(256), (size_t)0, stream, l.finite);
    }
    launch_pdl(kernel(l.half, l.p.term != nullptr, l.paired), dim3(l.grid), dim3(l.paired ? 320 : 192), (size_t)l.smem_bytes, stream, l.map_q, l.map_k, l.map_v, l.p);
    return (int)cudaGetLastError();
}

}  // namespace kn
