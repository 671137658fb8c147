// Exact-f32 contraction kernels on the SIMT pipes: batched matrix multiply and 2D convolution
// (as an implicit GEMM) with the fused `act(x + add1 + add2)` epilogue.
//
// These serve KN_MATH_F32 and every contraction shape the tensor-core kernels do not take
// (arbitrary operand strides, stride/padding combinations, tiny extents).  Operands are addressed
// through their element strides, so transposed, sliced, flipped or broadcast inputs need no copy.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <initializer_list>
#include <mutex>
#include <utility>

#include "../kernels.h"

#include "epilogue.cuh"
#include "launch.cuh"
#include "tc_ptx.cuh"

namespace kn {

namespace {

__device__ __forceinline__ float apply_epilogue(float v, int act, int round_tf32) {
    v = apply_activation(v, act);
    if (round_tf32) {
        uint32_t u;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v));
        v = __uint_as_float(u);
    }
    return v;
}

// ---------------------------------------------------------------- problems
// A problem tells the kernel where its operands are.  The reduction runs over `taps()` taps of `inner()` elements each
// (a matmul: one tap of k; a convolution: one tap per filter position, over the channels), so that inside a tap an
// operand is a pointer and a stride.  A `Tap` is what all rows and columns share about the current one.

struct OneTap {};

// Where a row of the A operand is, for the table that contract_cols_kernel keeps in shared memory: an element offset and,
// for a convolution, the window's first tap (kNoRow: the row does not exist).
struct RowAt { int64_t at; int iy, ix; };
constexpr int kNoRow = -(1 << 30);

struct GemmProblem {
    GemmParams p;
    using Element = float;
    using Tap = OneTap;
    __device__ int taps() const { return 1; }
    __device__ Tap tap(int) const { return Tap{}; }
    __device__ void next(Tap&) const {}
    __device__ int64_t inner() const { return p.k; }
    __device__ int64_t rows() const { return p.m; }
    __device__ int64_t cols() const { return p.n; }
    struct Row { const float* at; };
    __device__ Row row(int64_t b, int64_t m) const { return Row{p.a + b * p.sa[0] + m * p.sa[1]}; }
    __device__ const float* a_base() const { return p.a; }
    __device__ const float* a_at(const Row& r, const Tap&) const { return r.at; }
    __device__ int64_t a_stride() const { return p.sa[2]; }
    __device__ const float* col(int64_t b, int64_t n) const { return p.b + b * p.sb[0] + n * p.sb[2]; }
    __device__ const float* b_at(const float* col, const Tap&) const { return col; }
    __device__ int64_t b_stride() const { return p.sb[1]; }
    struct Out { int64_t b, m; };
    __device__ Out out(int64_t b, int64_t m) const { return Out{b, m}; }
    __device__ void store(const Out& o, int64_t n, float acc) const {
        if (p.add1) acc += p.add1[o.b * p.s1[0] + o.m * p.s1[1] + n * p.s1[2]];
        if (p.add2) acc += p.add2[o.b * p.s2[0] + o.m * p.s2[1] + n * p.s2[2]];
        p.c[o.b * p.sc[0] + o.m * p.sc[1] + n * p.sc[2]] = apply_epilogue(acc, p.act, p.round_tf32);
    }
    __device__ RowAt row_at(int64_t b, int64_t m) const { return RowAt{b * p.sa[0] + m * p.sa[1], 0, 0}; }
    __device__ bool inside(const RowAt&, const Tap&) const { return true; }
    __device__ int64_t tap_offset(const Tap&) const { return 0; }
    __device__ bool b_constant() const { return p.b_const != 0; }
    // where the result and the addends of a row are; their strides along the columns
    struct Line { int64_t o, a1, a2; };
    __device__ Line line(int64_t b, int64_t m) const {
        return Line{b * p.sc[0] + m * p.sc[1], b * p.s1[0] + m * p.s1[1], b * p.s2[0] + m * p.s2[1]};
    }
    __device__ float* result() const { return p.c; }
    __device__ int64_t result_stride() const { return p.sc[2]; }
    __device__ int64_t add1_stride() const { return p.s1[2]; }
    __device__ int64_t add2_stride() const { return p.s2[2]; }
};

// The same problem with f16 storage: operands and addends are converted on load, products accumulate in f32,
// the result is rounded to f16 once.
struct GemmProblemHalf {
    GemmParams p;
    using Element = __half;
    using Tap = OneTap;
    __device__ int taps() const { return 1; }
    __device__ Tap tap(int) const { return Tap{}; }
    __device__ void next(Tap&) const {}
    __device__ int64_t inner() const { return p.k; }
    __device__ int64_t rows() const { return p.m; }
    __device__ int64_t cols() const { return p.n; }
    struct Row { const __half* at; };
    __device__ Row row(int64_t b, int64_t m) const { return Row{(const __half*)p.a + b * p.sa[0] + m * p.sa[1]}; }
    __device__ const __half* a_base() const { return (const __half*)p.a; }
    __device__ const __half* a_at(const Row& r, const Tap&) const { return r.at; }
    __device__ int64_t a_stride() const { return p.sa[2]; }
    __device__ const __half* col(int64_t b, int64_t n) const { return (const __half*)p.b + b * p.sb[0] + n * p.sb[2]; }
    __device__ const __half* b_at(const __half* col, const Tap&) const { return col; }
    __device__ int64_t b_stride() const { return p.sb[1]; }
    struct Out { int64_t b, m; };
    __device__ Out out(int64_t b, int64_t m) const { return Out{b, m}; }
    __device__ void store(const Out& o, int64_t n, float acc) const {
        if (p.add1) acc += __half2float(((const __half*)p.add1)[o.b * p.s1[0] + o.m * p.s1[1] + n * p.s1[2]]);
        if (p.add2) acc += __half2float(((const __half*)p.add2)[o.b * p.s2[0] + o.m * p.s2[1] + n * p.s2[2]]);
        ((__half*)p.c)[o.b * p.sc[0] + o.m * p.sc[1] + n * p.sc[2]] = __float2half_rn(apply_activation(acc, p.act));
    }
};

struct ConvProblem {
    ConvParams p;
    using Element = float;
    struct Tap { int fy, fx; int64_t a, b; };
    __device__ int taps() const { return p.r * p.s; }
    __device__ Tap tap(int t) const {
        const int fy = t / p.s, fx = t - fy * p.s;
        return Tap{fy, fx, fy * p.s_in[2] + fx * p.s_in[3], fy * p.s_f[2] + fx * p.s_f[3]};
    }
    __device__ void next(Tap& t) const {
        t.fx++, t.a += p.s_in[3], t.b += p.s_f[3];
        if (t.fx == p.s) t.fx = 0, t.fy++, t.a += p.s_in[2] - p.s * p.s_in[3], t.b += p.s_f[2] - p.s * p.s_f[3];
    }
    __device__ int64_t inner() const { return p.c; }
    __device__ int64_t rows() const { return (int64_t)p.n * p.oh * p.ow; }
    __device__ int64_t cols() const { return p.k; }
    struct Row { const float* at; int iy, ix; };   // of the window's first tap, which may lie outside the image
    __device__ Row row(int64_t, int64_t m) const {
        const int64_t t = m / p.ow, img = t / p.oh;
        const int iy = (int)(t - img * p.oh) * p.stride_y - p.pad_y, ix = (int)(m - t * p.ow) * p.stride_x - p.pad_x;
        return Row{p.in + img * p.s_in[0] + iy * p.s_in[2] + ix * p.s_in[3], iy, ix};
    }
    __device__ const float* a_base() const { return p.in; }
    __device__ const float* a_at(const Row& r, const Tap& t) const {   // null outside the image
        return (unsigned)(r.iy + t.fy) < (unsigned)p.h && (unsigned)(r.ix + t.fx) < (unsigned)p.w ? r.at + t.a : nullptr;
    }
    __device__ int64_t a_stride() const { return p.s_in[1]; }
    __device__ const float* col(int64_t, int64_t n) const { return p.filter + n * p.s_f[0]; }
    __device__ const float* b_at(const float* col, const Tap& t) const { return col + t.b; }
    __device__ int64_t b_stride() const { return p.s_f[1]; }
    struct Out { int64_t o, a1, a2; };
    __device__ Out out(int64_t, int64_t m) const {
        const int64_t t = m / p.ow, img = t / p.oh, ox = m - t * p.ow, oy = t - img * p.oh;
        return Out{img * p.s_out[0] + oy * p.s_out[2] + ox * p.s_out[3], img * p.s1[0] + oy * p.s1[2] + ox * p.s1[3],
                   img * p.s2[0] + oy * p.s2[2] + ox * p.s2[3]};
    }
    __device__ void store(const Out& o, int64_t n, float acc) const {
        if (p.add1) acc += p.add1[o.a1 + n * p.s1[1]];
        if (p.add2) acc += p.add2[o.a2 + n * p.s2[1]];
        p.out[o.o + n * p.s_out[1]] = apply_epilogue(acc, p.act, p.round_tf32);
    }
    __device__ RowAt row_at(int64_t b, int64_t m) const {
        const Row r = row(b, m);
        return RowAt{r.at - p.in, r.iy, r.ix};
    }
    __device__ bool inside(const RowAt& r, const Tap& t) const { return (unsigned)(r.iy + t.fy) < (unsigned)p.h && (unsigned)(r.ix + t.fx) < (unsigned)p.w; }
    __device__ int64_t tap_offset(const Tap& t) const { return t.a; }
    __device__ bool b_constant() const { return p.f_const != 0; }
    using Line = Out;
    __device__ Line line(int64_t b, int64_t m) const { return out(b, m); }
    __device__ float* result() const { return p.out; }
    __device__ int64_t result_stride() const { return p.s_out[1]; }
    __device__ int64_t add1_stride() const { return p.s1[1]; }
    __device__ int64_t add2_stride() const { return p.s2[1]; }
};

// ---------------------------------------------------------------- the kernel
constexpr int kThreads = 256, BK = 32, kStages = 3;
constexpr int TM = 8;            // rows per thread
constexpr int kTilePad = 4;      // row padding of the partial result tile

// Shared tiles are [row][K], K contiguous, rows padded by 16 bytes: the 128-bit reads of eight neighbouring rows then
// cover all banks once.
template <class E> constexpr int row_elements = BK + 16 / (int)sizeof(E);
template <class E, int BM, int BN> constexpr int stage_bytes = (BM + BN) * row_elements<E> * (int)sizeof(E);
template <int BM, int BN, int KG> constexpr int tile_bytes = KG * BM * (BN + kTilePad) * 4;
template <class E, int BM, int BN, int KG>
constexpr int smem_bytes = kStages * stage_bytes<E, BM, BN> > tile_bytes<BM, BN, KG> ? kStages * stage_bytes<E, BM, BN> : tile_bytes<BM, BN, KG>;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// `bytes` (0 .. 16) bytes of global memory, zeros up to 16
__device__ __forceinline__ void fetch16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// one element, or a zero (`src` is a valid address either way)
__device__ __forceinline__ void fetch1(float* dst, const float* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void fetch1(__half* dst, const __half* src, bool in) { *dst = in ? *src : __float2half_rn(0.f); }

// four K elements of a row
__device__ __forceinline__ float4 read4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 read4(const __half* p) {
    const uint2 h = *(const uint2*)p;
    const float2 lo = __half22float2(*(const __half2*)&h.x), hi = __half22float2(*(const __half2*)&h.y);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

enum class Load : int { Wide, AlongK, AlongRows };   // how an operand is fetched: 16 bytes along K; one element along K / along its rows
struct TileArgs {
    int slices;              // of K, one cluster
    Load load_a, load_b;
    bool rows_fast;          // the result's rows, not its columns, are contiguous
};

// C tile of BM x BN per CTA, 8 x TN per thread, KG thread groups taking alternate halves of a K block (summed in shared
// memory at the end).  `gridDim.z` = batch x slices of K; the slices of a tile are one cluster and sum their tiles
// through distributed shared memory, so a problem with few tiles still fills the chip and needs no second launch.
//
// What bounds it is instruction issue.  Operands arrive 16 bytes at a time and stay along K in shared memory; four K
// elements cost a thread 32 TN multiply-adds next to 8 + TN 128-bit reads.  (With the tiles along their rows, as the
// classic layout has it, elements arrived by 4-byte copies, whose addresses were most of the instructions: 127 us
// for 4096 positions x 128 channels x 1152, against 345 us of the kernel before it.)
//   128 x 128, 8 x 8 per thread       the fewest reads per multiply-add; for problems that fill the chip with such tiles
//    64 x  64, 8 x 4 per thread, KG 2  four times the tiles
// Plain multiply-adds: the packed form (fma.rn.f32x2) issues at half the rate and measured 5 % slower, K blocks of 64
// spilled registers.  4096 positions x 128 channels x 1152: 48 to 52 us
// (36 by contract_cols_kernel, which kernel_bench's conv_exact takes now); 19200 x 256 x 2304: 800 us (two tiles a SM, three
// rounds of 148 for 300 tiles).
// `Index` counts along K: 64 bits for reductions that 32 do not hold.
template <class Problem, int BM, int BN, int TN, int KG, class Index>
__global__ void __launch_bounds__(kThreads, KG) contract_simt_kernel(const __grid_constant__ Problem prob, const __grid_constant__ TileArgs args) {
    constexpr int TX = BN / TN, TY = BM / TM;
    static_assert(TX * TY * KG == kThreads, "one output tile per CTA");
    using E = typename Problem::Element;
    constexpr int LR = row_elements<E>, kWide = 16 / (int)sizeof(E);
    extern __shared__ __align__(16) uint8_t smem[];
    pdl_enter();
    const int slices = args.slices;
    const int64_t M = prob.rows(), N = prob.cols();
    const Index inner = (Index)prob.inner();
    const int taps = prob.taps();
    const int slice = (int)(blockIdx.z % (unsigned)slices);
    const int64_t batch = blockIdx.z / (unsigned)slices;
    const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
    const int tid = threadIdx.x;
    const int group = tid / (TX * TY), rank = tid % (TX * TY);
    // Which rows and columns a lane takes decides what its 128-bit shared reads cost: half a warp's are served in one pass
    // if lanes i and i ^ 1 (or i and i ^ 2) all read the same address, else in two.  Bit 0 and bit 4 of the lane pick the
    // column, bits 1 to 3 the row: both operands' reads qualify (with rows along bits 0 to 2 an operand's did not:
    // 40 passes per four K elements instead of 24, and the reads, not the multiply-adds, were the limit).
    const int warp = rank >> 5, lane = rank & 31;
    const int ty = ((lane >> 1) & 7) + 8 * (warp % (TY / 8)), tx = ((lane & 1) | ((lane >> 4) << 1)) + 4 * (warp / (TY / 8));

    // K blocks of this slice: block kb is elements (kb % per_tap) * BK .. of tap kb / per_tap
    // (an empty reduction has none: the result is the addends)
    const Index per_tap = max((Index)1, (inner + BK - 1) / BK);
    const Index total = inner > 0 ? taps * per_tap : 0, per_slice = (total + slices - 1) / slices;
    const Index kb_first = min(slice * per_slice, total), blocks = min(kb_first + per_slice, total) - kb_first;

    // 16-byte fetches: chunk tid % (BK / kWide) of rows tid / (BK / kWide) + i * kRowStep
    constexpr int kChunks = BK / kWide, kRowStep = kThreads / kChunks;
    constexpr int A_ROWS = BM / kRowStep > 0 ? BM / kRowStep : 1, B_ROWS = BN / kRowStep > 0 ? BN / kRowStep : 1;
    const int chunk = tid % kChunks, chunk_row = tid / kChunks;
    typename Problem::Row a_rows[A_ROWS];
    uint32_t a_valid = 0;
    if (args.load_a == Load::Wide) {
#pragma unroll
        for (int i = 0; i < A_ROWS; i++) {
            const int mm = chunk_row + i * kRowStep;
            const bool in = mm < BM && m0 + mm < M;
            a_valid |= (uint32_t)in << i;
            a_rows[i] = prob.row(batch, in ? m0 + mm : 0);
        }
    }
    // An address to name where nothing is read.  cp.async wants its source aligned to the copy's size even then, so each
    // operand names its own base: the other one may start at any element.
    const E* const no_a = prob.a_base();
    const E* const no_b = prob.col(0, 0);
    int load_tap = (int)(kb_first / per_tap);
    Index load_block = kb_first - load_tap * per_tap;
    typename Problem::Tap tap = prob.tap(load_tap);
    const E* a_at[A_ROWS];
    const E* b_at[B_ROWS];
    const E* b_col[B_ROWS];
    uint32_t a_read = 0, b_read = 0;   // rows and columns that exist (and, for a row, whose window is inside the image)
#pragma unroll
    for (int i = 0; i < B_ROWS; i++) {
        const int nn = chunk_row + i * kRowStep;
        const bool in = args.load_b == Load::Wide && nn < BN && n0 + nn < N;
        b_col[i] = in ? prob.col(batch, n0 + nn) : no_b;
        b_read |= (uint32_t)in << i;
    }
    auto enter_tap = [&] {
        a_read = 0;
        const Index k0 = load_block * BK + chunk * kWide;
        if (args.load_a == Load::Wide) {
#pragma unroll
            for (int i = 0; i < A_ROWS; i++) {
                const E* at = ((a_valid >> i) & 1) ? prob.a_at(a_rows[i], tap) : nullptr;
                a_read |= (uint32_t)(at != nullptr) << i;
                a_at[i] = at ? at + k0 : no_a;
            }
        }
#pragma unroll
        for (int i = 0; i < B_ROWS; i++) b_at[i] = ((b_read >> i) & 1) ? prob.b_at(b_col[i], tap) + k0 : no_b;
    };
    enter_tap();
    const uint32_t fetch_to = smem_addr(smem) + (uint32_t)(chunk_row * LR + chunk * kWide) * (uint32_t)sizeof(E);
    auto load_stage = [&](int stage) {
        const uint32_t to = fetch_to + (uint32_t)stage * stage_bytes<E, BM, BN>;
        const Index k0 = load_block * BK;
        const Index left = inner - k0 - chunk * kWide;   // elements of the row from this chunk on
        const int bytes = (int)min((Index)kWide, max((Index)0, left)) * (int)sizeof(E);
        if (args.load_a == Load::Wide) {
#pragma unroll
            for (int i = 0; i < A_ROWS; i++) {
                if (BM % kRowStep == 0 || chunk_row + i * kRowStep < BM)
                    fetch16(to + i * kRowStep * LR * (int)sizeof(E), left > 0 ? a_at[i] : no_a, ((a_read >> i) & 1) ? bytes : 0);
                a_at[i] += ((a_read >> i) & 1) ? BK : 0;
            }
        } else {
            E* As = (E*)(smem + stage * stage_bytes<E, BM, BN>);
            const bool along_k = args.load_a == Load::AlongK;
#pragma unroll 1
            for (int e = tid; e < BM * BK; e += kThreads) {
                const int mm = along_k ? e / BK : e % BM, kk = along_k ? e % BK : e / BM;
                const E* src = nullptr;
                if (m0 + mm < M && k0 + kk < inner) src = prob.a_at(prob.row(batch, m0 + mm), tap);
                fetch1(As + mm * LR + kk, src ? src + (k0 + kk) * prob.a_stride() : no_a, src != nullptr);
            }
        }
        if (args.load_b == Load::Wide) {
#pragma unroll
            for (int i = 0; i < B_ROWS; i++) {
                if (BN % kRowStep == 0 || chunk_row + i * kRowStep < BN)
                    fetch16(to + (BM + i * kRowStep) * LR * (int)sizeof(E), left > 0 ? b_at[i] : no_b, ((b_read >> i) & 1) ? bytes : 0);
                b_at[i] += ((b_read >> i) & 1) ? BK : 0;
            }
        } else {
            E* Bs = (E*)(smem + stage * stage_bytes<E, BM, BN>) + BM * LR;
            const bool along_k = args.load_b == Load::AlongK;
#pragma unroll 1
            for (int e = tid; e < BN * BK; e += kThreads) {
                const int nn = along_k ? e / BK : e % BN, kk = along_k ? e % BK : e / BN;
                const bool in = n0 + nn < N && k0 + kk < inner;
                fetch1(Bs + nn * LR + kk, in ? prob.b_at(prob.col(batch, n0 + nn), tap) + (k0 + kk) * prob.b_stride() : no_b, in);
            }
        }
        if (++load_block == per_tap) {
            load_block = 0;
            if (++load_tap < taps) {
                prob.next(tap);
                enter_tap();
            }
        }
    };

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;

#pragma unroll
    for (int s = 0; s < kStages - 1; s++) {
        if (s < blocks) load_stage(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0, next = kStages - 1;
#pragma unroll 1
    for (Index b = 0; b < blocks; b++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();   // stage `b` is complete, and everybody has read stage `b - 1`, which is filled next
        if (b + kStages - 1 < blocks) load_stage(next);
        asm volatile("cp.async.commit_group;" ::: "memory");
        // a thread's rows are TY (its columns TX) apart: neighbouring lanes read neighbouring rows
        const E* As = (const E*)(smem + stage * stage_bytes<E, BM, BN>) + ty * LR + group * (BK / KG);
        const E* Bs = (const E*)(smem + stage * stage_bytes<E, BM, BN>) + (BM + tx) * LR + group * (BK / KG);
#pragma unroll
        for (int k = 0; k < BK / KG; k += 4) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; j++) w[j] = read4(Bs + j * TX * LR + k);
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const float4 a = read4(As + i * TY * LR + k);
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
            }
        }
        if (++stage == kStages) stage = 0;
        if (++next == kStages) next = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // the tile (one per thread group) in shared memory, [KG][BM][BN + pad]; read back along the result's contiguous axis
    constexpr int LC = BN + kTilePad, kTile = BM * LC;
    float* tile = (float*)smem;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) tile[group * kTile + (ty + i * TY) * LC + tx + j * TX] = acc[i][j];
    if (slices > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    const uint32_t own = smem_addr(tile);
    for (int e = slice * kThreads + tid; e < BM * BN; e += slices * kThreads) {
        const int mm = args.rows_fast ? e % BM : e / BN, nn = args.rows_fast ? e / BM : e % BN;
        const int64_t m = m0 + mm, n = n0 + nn;
        if (m >= M || n >= N) continue;
        float v = 0.f;
        for (int q = 0; q < slices; q++) {
            uint32_t from = own;
            if (slices > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(own), "r"(q));
#pragma unroll
            for (int g = 0; g < KG; g++) {
                float x;
                const uint32_t at = from + 4u * (uint32_t)(g * kTile + mm * LC + nn);
                if (slices > 1) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at));
                else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(at));
                v += x;
            }
        }
        prob.store(prob.out(batch, m), n, v);
    }
    if (slices > 1) {   // nobody leaves while a peer still reads its tile
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// ---------------------------------------------------------------- B along its columns
// The kernel for operands B whose columns, not whose reduction, are contiguous: V of an attention step as it comes, and the
// filters and weights that the planner lays out this way (plan.cpp: `filter_rows`).
//
// A tile of B is [K][columns] in shared memory, so two neighbouring columns of a thread are one 64-bit operand of a packed
// multiply-add (fma.rn.f32x2) whose other factor is one element of A twice: half the instructions of plain multiply-adds and
// no pair of operands in one register bank.  Tiles along K (contract_simt_kernel above) cannot have that without twice the
// accumulators.  A matmul of 16384 x 1024 x 2048: 0.73 of 74.4 TFLOP/s (the chip's own limit for either form at the clocks it
// holds is 70 to 72) against 0.66.
//    64 x 64, 8 x 8 per thread, two groups, 128 threads, three CTAs per SM: the registers allow no more, and twelve warps an
//             SM hide the shared reads that eight of a 128 x 128 tile do not (equal where those fill the chip, 0.66 against
//             0.56 where they do not)
//    the same with four groups, 256 threads, where at most 148 CTAs of it come out cheapest: no slower than two groups in 44 of
//             45 matmuls and convolutions, 4 % slower in one (639 x 127 x 2077: 41.3 us, 39.6), and closer to 64 bits (sums over a
//             quarter of a K block)
//    32 x 32, 4 x 4 per thread, four groups: for problems of a few tiles, where it is the number of CTAs that counts
// What a small problem costs is latency, so: the constant operand is requested ahead of the dependency wait, for as many
// stages as there are; rows are located once, in a table, and not by divisions in the loop; slices of a tile send their sums to
// the CTA that stores them (a cluster barrier that the peers have started, waited for at the first remote store; no remote reads).
// COUNTED: that they have arrived is told by a barrier in the receiver's memory that counts their bytes (`st.async`), not by a
// second cluster barrier, which has to release what it hands over and takes some 1000 cycles.  Not where three and more large tiles
// share an SM, another CTA computing meanwhile, or eight slices do: the code with the counter is the slower one there, even
// without slices (seven layers of 128 channels: 40 boards 178 -> 186 us with it, 95 373 -> 381, 256 715 -> 722; eight boards of 256
// channels 102 -> 106; with two tiles an SM two batches of 22 boards at a time 1009 -> 988 for 33 layers).
// One 8 x 8 board, 128 -> 128 channels, 3 x 3: 12.1 us on contract_simt_kernel, 5.2 us here (5.6 with a second cluster barrier)
// (in a chain; by itself 7.4, kernel_bench's conv_exact_board); 64 boards 48 -> 36 us, 256 boards 112 us
// (0.61 of the rate); 12 heads of 120 x 64 x 120 (probabilities . V) 14.1 -> 4.8 us.
template <int BM, int BN, int TM, int TN, int KG, int ST>
struct ColsLayout {
    static constexpr int kThreads = BM / TM * (BN / TN) * KG;
    static constexpr int kPitchA = BK + 4, kBytesA = BM * kPitchA * 4, kStage = kBytesA + BK * BN * 4;
    static constexpr int kPitchC = BN + 4, kTile = KG * BM * kPitchC * 4;
    static constexpr int kFront = ST * kStage > kTile ? ST * kStage : kTile;   // stages, then (in their place) the partial tiles
    static constexpr int kUnits = BM * BN / 4;                                  // groups of four columns
    static constexpr int kReceived = (kUnits + 8) * 16;                         // sums sent by the other slices
    static constexpr int kBarrier = kFront + kReceived + BM * (int)sizeof(RowAt) + BM * 24;   // counts the bytes of sums that arrive
    static constexpr int kBytes = kBarrier + 16;
};

struct ColsArgs {
    int slices;
    Load load_a;
    bool wide_b;      // 16-byte fetches of B
    bool rows_fast;   // the result's rows, not its columns, are contiguous
    bool wide_c;      // four columns of the result are one aligned 16-byte store
};

template <class Problem, int BM, int BN, int TM, int TN, int KG, int ST, int OCC, bool COUNTED>
__global__ void __launch_bounds__(BM / TM * (BN / TN) * KG, OCC)
contract_cols_kernel(const __grid_constant__ Problem prob, const __grid_constant__ ColsArgs args) {
    using L = ColsLayout<BM, BN, TM, TN, KG, ST>;
    constexpr int TX = BN / TN, TY = BM / TM, NT = L::kThreads;
    static_assert(TX % 4 == 0 && TY % 8 == 0 && TN % 4 == 0, "lane layout");
    extern __shared__ __align__(16) uint8_t smem[];
    float4* const received = (float4*)(smem + L::kFront);
    RowAt* const rows = (RowAt*)(smem + L::kFront + L::kReceived);
    typename Problem::Line* const lines = (typename Problem::Line*)(rows + BM);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int slices = args.slices;
    const int slice = (int)(blockIdx.z % (unsigned)slices);
    // units of four columns of the result, of which each slice stores `share`
    int share = 0;
    if (COUNTED) share = (L::kUnits + slices - 1) / slices;
    const uint32_t arrived = smem_addr(smem + L::kBarrier);
    if (slices > 1) {
        if (COUNTED) {
            if (threadIdx.x == 0) {
                tcp::mbar_init(arrived, 1);
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                tcp::mbar_expect_tx(arrived, (uint32_t)(max(0, min(share, L::kUnits - slice * share)) * slices) * 16u);
            }
            __syncwarp();
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (waited for before the first remote store)
    }
    const int64_t M = prob.rows(), N = prob.cols();
    const int inner = (int)prob.inner(), taps = prob.taps();
    const int64_t batch = blockIdx.z / (unsigned)slices;
    const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
    const int tid = threadIdx.x;

    const int per_tap = max(1, (inner + BK - 1) / BK);
    const int total = inner > 0 ? taps * per_tap : 0, per_slice = (total + slices - 1) / slices;
    const int kb_first = min(slice * per_slice, total), blocks = min(kb_first + per_slice, total) - kb_first;

    // B: row kk of a K block is row (tap, block * BK + kk) of the operand
    constexpr int kChunksB = BN / 4, kRowStepB = NT / kChunksB, kRowsB = BK / kRowStepB;
    static_assert(NT % kChunksB == 0 && BK % kRowStepB == 0 && NT % 8 == 0 && BM % (NT / 8) == 0, "fetch layout");
    const int64_t b_stride = prob.b_stride();
    const float* const b_first = prob.col(batch, n0);
    const int b_chunk = tid % kChunksB, b_row = tid / kChunksB;
    const int b_bytes = (int)max((int64_t)0, min((int64_t)4, N - n0 - b_chunk * 4)) * 4;
    auto load_b = [&](int stage, const typename Problem::Tap& tap, int block) {
        float* Bs = (float*)(smem + stage * L::kStage + L::kBytesA);
        const int left = inner - block * BK;
        const float* src = prob.b_at(b_first, tap) + (int64_t)block * BK * b_stride;
        if (args.wide_b) {
            const float* at = src + b_row * b_stride + b_chunk * 4;
            const uint32_t to = smem_addr(Bs + b_row * BN + b_chunk * 4);
#pragma unroll
            for (int i = 0; i < kRowsB; i++) {
                const bool in = b_row + i * kRowStepB < left && b_bytes > 0;
                fetch16(to + i * kRowStepB * BN * 4, in ? at + (int64_t)i * kRowStepB * b_stride : b_first, in ? b_bytes : 0);
            }
        } else {
#pragma unroll 4
            for (int e = tid; e < BK * BN; e += NT) {
                const int kk = e / BN, nn = e % BN;
                const bool in = kk < left && n0 + nn < N;
                fetch1(Bs + e, in ? src + kk * b_stride + nn : b_first, in);
            }
        }
    };
    int load_tap = kb_first / per_tap, load_block = kb_first - load_tap * per_tap;   // what load_a fetches next
    typename Problem::Tap tap = prob.tap(load_tap);
    const bool early_b = prob.b_constant();
    if (early_b) {
        int t = load_tap, block = load_block;
        typename Problem::Tap at = tap;
        for (int s = 0; s < ST - 1 && s < blocks; s++) {
            load_b(s, at, block);
            if (++block == per_tap) {
                block = 0;
                if (++t < taps) prob.next(at);
            }
        }
    }
    for (int i = tid; i < BM; i += NT) {
        const bool in = m0 + i < M;
        rows[i] = in ? prob.row_at(batch, m0 + i) : RowAt{0, kNoRow, 0};
        lines[i] = prob.line(batch, in ? m0 + i : 0);
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // A, 16-byte fetches: chunk tid % 8 of rows tid / 8 + i * kRowStepA
    constexpr int kRowStepA = NT / 8, kRowsA = BM / kRowStepA;
    const float* const a_base = prob.a_base();
    const int a_chunk = tid % 8, a_row = tid / 8;
    const float* a_at[kRowsA];
    uint32_t a_read = 0;
    auto enter_tap = [&] {
        a_read = 0;
        if (args.load_a != Load::Wide) return;
        const int64_t offset = prob.tap_offset(tap) + load_block * BK + a_chunk * 4;
#pragma unroll
        for (int i = 0; i < kRowsA; i++) {
            const RowAt r = rows[a_row + i * kRowStepA];
            const bool in = r.iy != kNoRow && prob.inside(r, tap);
            a_read |= (uint32_t)in << i;
            a_at[i] = in ? a_base + r.at + offset : a_base;
        }
    };
    enter_tap();
    auto load_a = [&](int stage) {
        float* As = (float*)(smem + stage * L::kStage);
        const int k0 = load_block * BK;
        if (args.load_a == Load::Wide) {
            const int left = inner - k0 - a_chunk * 4, bytes = min(4, max(0, left)) * 4;
            const uint32_t to = smem_addr(As + a_row * L::kPitchA + a_chunk * 4);
#pragma unroll
            for (int i = 0; i < kRowsA; i++) {
                const bool in = (a_read >> i) & 1;
                fetch16(to + i * kRowStepA * L::kPitchA * 4, left > 0 ? a_at[i] : a_base, in ? bytes : 0);
                a_at[i] += in ? BK : 0;
            }
        } else {
            const bool along_k = args.load_a == Load::AlongK;
            const int64_t stride = prob.a_stride(), offset = prob.tap_offset(tap) + k0 * stride;
#pragma unroll 4
            for (int e = tid; e < BM * BK; e += NT) {
                const int mm = along_k ? e / BK : e % BM, kk = along_k ? e % BK : e / BM;
                const RowAt r = rows[mm];
                const bool in = r.iy != kNoRow && k0 + kk < inner && prob.inside(r, tap);
                fetch1(As + mm * L::kPitchA + kk, in ? a_base + r.at + offset + kk * stride : a_base, in);
            }
        }
    };
    auto advance = [&] {
        if (++load_block == per_tap) {
            load_block = 0;
            if (++load_tap < taps) {
                prob.next(tap);
                enter_tap();
            }
        }
    };

    const int group = tid / (TX * TY), rank = tid % (TX * TY), warp = rank >> 5, lane = rank & 31;
    // (which lanes share rows and columns: see contract_simt_kernel)
    const int tx = ((lane & 1) | ((lane >> 4) << 1)) + 4 * (warp % (TX / 4)), ty = ((lane >> 1) & 7) + 8 * (warp / (TX / 4));
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = make_float2(0.f, 0.f);

#pragma unroll 1
    for (int s = 0; s < ST - 1; s++) {
        if (s < blocks) {
            if (!early_b) load_b(s, tap, load_block);
            load_a(s);
            advance();
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0, next = ST - 1;
#pragma unroll 1
    for (int b = 0; b < blocks; b++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();   // stage `b` is complete, and everybody has read stage `b - 1`, which is filled next
        if (b + ST - 1 < blocks) {
            load_b(next, tap, load_block);
            load_a(next);
            advance();
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* As = (const float*)(smem + stage * L::kStage) + ty * L::kPitchA + group * (BK / KG);
        const float* Bs = (const float*)(smem + stage * L::kStage + L::kBytesA) + group * (BK / KG) * BN + tx * 4;
#pragma unroll
        for (int k = 0; k < BK / KG; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = read4(As + i * TY * L::kPitchA + k);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float4 w[TN / 4];
#pragma unroll
                for (int j = 0; j < TN / 4; j++) w[j] = read4(Bs + (k + q) * BN + j * TX * 4);
#pragma unroll
                for (int i = 0; i < TM; i++) {
                    const float x = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
#pragma unroll
                    for (int j = 0; j < TN / 4; j++) {
                        acc[i][2 * j] = fma_pair(make_float2(x, x), make_float2(w[j].x, w[j].y), acc[i][2 * j]);
                        acc[i][2 * j + 1] = fma_pair(make_float2(x, x), make_float2(w[j].z, w[j].w), acc[i][2 * j + 1]);
                    }
                }
            }
        }
        if (++stage == ST) stage = 0;
        if (++next == ST) next = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // the tile, one per thread group, in shared memory: [KG][BM][BN + 4]
    float* tile = (float*)smem;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 4; j++)
            *(float4*)(tile + (group * BM + ty + i * TY) * L::kPitchC + (j * TX + tx) * 4) =
                make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
    __syncthreads();
    if (slices > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // units, in the order in which the result's contiguous axis comes first
    if (!COUNTED) share = (L::kUnits + slices - 1) / slices;
    auto place = [&](int u, int& mm, int& nn) {
        mm = args.rows_fast ? u % BM : u / (BN / 4);
        nn = (args.rows_fast ? u / BM : u % (BN / 4)) * 4;
    };
    float* const result = prob.result();
    const int64_t c_stride = prob.result_stride(), s1 = prob.add1_stride(), s2 = prob.add2_stride();
    auto store = [&](int mm, int nn, float4 v) {
        if (m0 + mm >= M) return;
        const typename Problem::Line l = lines[mm];
        float x[4] = {v.x, v.y, v.z, v.w};
        const int64_t n = n0 + nn;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (n + i >= N) break;
            if (prob.p.add1) x[i] += prob.p.add1[l.a1 + (n + i) * s1];
            if (prob.p.add2) x[i] += prob.p.add2[l.a2 + (n + i) * s2];
            x[i] = apply_epilogue(x[i], prob.p.act, prob.p.round_tf32);
            if (!args.wide_c) result[l.o + (n + i) * c_stride] = x[i];
        }
        if (args.wide_c && n < N) *(float4*)(result + l.o + n) = make_float4(x[0], x[1], x[2], x[3]);
    };
    for (int u = tid; u < L::kUnits; u += NT) {
        int mm, nn;
        place(u, mm, nn);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int g = 0; g < KG; g++) {
            const float4 t = *(const float4*)(tile + (g * BM + mm) * L::kPitchC + nn);
            v.x += t.x, v.y += t.y, v.z += t.z, v.w += t.w;
        }
        if (slices == 1) {
            store(mm, nn, v);
        } else {
            const int owner = u / share;
            const uint32_t to = tcp::map_to_cta(smem_addr(received + slice * share + u - owner * share), (uint32_t)owner);
            if constexpr (COUNTED)
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                             ::"r"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(tcp::map_to_cta(arrived, (uint32_t)owner))
                             : "memory");
            else
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
        }
    }
    if (slices > 1) {
        if constexpr (COUNTED) {
            const long long start = clock64();
            while (!tcp::mbar_try_wait_cluster(arrived, 0)) {
                if (clock64() - start > tcp::kWaitCycles) {
                    atomicMax(prob.p.status, 71u);
                    return;
                }
            }
        } else {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        for (int u = tid; u < share && slice * share + u < L::kUnits; u += NT) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int q = 0; q < slices; q++) {
                const float4 t = received[q * share + u];
                v.x += t.x, v.y += t.y, v.z += t.z, v.w += t.w;
            }
            int mm, nn;
            place(slice * share + u, mm, nn);
            store(mm, nn, v);
        }
    }
}

template <class Problem, int BM, int BN, int TM, int TN, int KG, int ST, int OCC, bool COUNTED>
int launch_cols_tile(const Problem& prob, int64_t M, int64_t N, int64_t batch, const ColsArgs& args, int at_least, cudaStream_t stream) {
    using L = ColsLayout<BM, BN, TM, TN, KG, ST>;
    auto kernel = contract_cols_kernel<Problem, BM, BN, TM, TN, KG, ST, OCC, COUNTED>;
    static std::mutex mu;
    static bool done[64] = {false};
    const int smem = std::max(L::kBytes, at_least);
    if (int e = allow_shared(kernel, std::max(L::kBytes, 80 * 1024), done, mu)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((M + BM - 1) / BM), (unsigned)((N + BN - 1) / BN), (unsigned)(batch * args.slices));
    cfg.blockDim = dim3(L::kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)args.slices;
    cfg.attrs = attr;
    cfg.numAttrs = args.slices > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, prob, args);
}

// Can contract_cols_kernel take the problem: as many tiles as the grid holds, K blocks that 32 bits count
bool cols_fits(int64_t M, int64_t N, int64_t batch, int64_t k_blocks) {
    return k_blocks < (1 << 25) && (N + 31) / 32 <= 65535 && batch * 8 <= 65535 && (M + 31) / 32 <= 0x7FFFFFFFll;
}

template <class Problem>
int launch_cols(const Problem& prob, int64_t M, int64_t N, int64_t batch, int64_t k_blocks, ColsArgs args, cudaStream_t stream) {
    if (M == 0 || N == 0 || batch == 0) return 0;
    // The tile and the number of slices whose busiest SM is done first: n CTAs of it, at the cycles that a K block and a CTA
    // were measured to take when several (or one) share an SM.
    enum { kLarge, kLargeAlone, kSmall } tile = kSmall;
    int64_t best = INT64_MAX, per_sm = 1;
    auto consider = [&](decltype(tile) t, int64_t tiles, int64_t slices) {
        const int64_t n = (tiles * slices + 147) / 148, blocks = (k_blocks + slices - 1) / slices;
        const int64_t block = t == kLarge ? (n <= 2 ? 1650 : 1550) : t == kLargeAlone ? 1900 : (n == 1 ? 900 : 650);
        const int64_t cost = n * (block * blocks + 700) + (slices > 1 ? 1500 : 0);
        if (cost < best) best = cost, tile = t, args.slices = (int)slices, per_sm = n;
    };
    const int64_t large = ((M + 63) / 64) * ((N + 63) / 64) * batch, small = ((M + 31) / 32) * ((N + 31) / 32) * batch;
    for (int64_t slices = 1; slices <= 8 && (slices == 1 || k_blocks >= 4 * slices); slices++) {
        consider(kSmall, small, slices);
        consider(large * slices <= 148 ? kLargeAlone : kLarge, large, slices);
    }
    if (tile == kSmall) return launch_cols_tile<Problem, 32, 32, 4, 4, 4, 6, 2, true>(prob, M, N, batch, args, 0, stream);
    if (tile == kLargeAlone) return launch_cols_tile<Problem, 64, 64, 8, 8, 4, 3, 1, true>(prob, M, N, batch, args, 0, stream);
    // (two CTAs an SM are kept at two by the shared memory they ask for: three on some SMs and one on others took 81 us
    // instead of 57 for 1024 x 1024 x 1024)
    if (per_sm <= 2 && args.slices < 8) return launch_cols_tile<Problem, 64, 64, 8, 8, 2, 3, 3, true>(prob, M, N, batch, args, 80 * 1024, stream);
    return launch_cols_tile<Problem, 64, 64, 8, 8, 2, 3, 3, false>(prob, M, N, batch, args, per_sm <= 2 ? 80 * 1024 : 0, stream);
}

template <class Problem, int BM, int BN, int TN, int KG, class Index = int>
int launch_tile(const Problem& prob, int64_t gx, int64_t gy, int64_t batch, const TileArgs& args, cudaStream_t stream) {
    auto kernel = contract_simt_kernel<Problem, BM, BN, TN, KG, Index>;
    constexpr int smem = smem_bytes<typename Problem::Element, BM, BN, KG>;
    static std::mutex mu;
    static bool done[64] = {false};
    if (int e = allow_shared(kernel, smem, done, mu)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)gx, (unsigned)gy, (unsigned)(batch * args.slices));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)args.slices;
    cfg.attrs = attr;
    cfg.numAttrs = args.slices > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, prob, args);
}

// `taps` x `inner`: the reduction
template <class Problem>
int launch(const Problem& prob, int64_t M, int64_t N, int64_t batch, int64_t taps, int64_t inner, TileArgs args, cudaStream_t stream) {
    if (M == 0 || N == 0 || batch == 0) return 0;
    const int64_t k_blocks = taps * ((inner + BK - 1) / BK);
    const int64_t large = ((M + 127) / 128) * ((N + 127) / 128) * batch, small = ((M + 63) / 64) * ((N + 63) / 64) * batch;
    // Rounds of tiles over the chip, times the time of a round: a 128 x 128 tile alone on its SM runs at 0.56 of the
    // multiply-add rate, two 64 x 64 tiles sharing one at 0.45 (both measured), and the last round may be nearly empty.
    const double rounds_large = (double)((large + 147) / 148) * 4 / 0.56, rounds_small = (double)((small + 295) / 296) * 2 / 0.45;
    const bool long_k = k_blocks > (1ll << 25);   // (the counters run one K block past the end)
    const bool wide = !long_k && rounds_large < rounds_small;
    const int64_t gx = (M + (wide ? 127 : 63)) / (wide ? 128 : 64), gy = (N + (wide ? 127 : 63)) / (wide ? 128 : 64);
    if (gy > 65535 || batch > 65535 || gx > 0x7FFFFFFFll) return (int)cudaErrorInvalidValue;
    args.slices = 1;
    if (wide) return launch_tile<Problem, 128, 128, 8, 1>(prob, gx, gy, batch, args, stream);
    // slices of K until the chip has two CTAs per SM (one alone leaves the schedulers two warps each, which cover neither
    // the shared reads nor the multiply-adds' latency), at least four blocks each (a slice pays the pipeline's fill and
    // two cluster barriers, some 3 us), eight at most (the portable cluster size)
    while (args.slices < 8 && gx * gy * batch * args.slices * 2 <= 296 && k_blocks >= 4 * 2 * args.slices && batch * args.slices * 2 <= 65535)
        args.slices *= 2;
    if (long_k) return launch_tile<Problem, 64, 64, 4, 2, int64_t>(prob, gx, gy, batch, args, stream);
    return launch_tile<Problem, 64, 64, 4, 2>(prob, gx, gy, batch, args, stream);
}

// 16-byte fetches along K: K contiguous, everything else a multiple of 16 bytes apart
Load load_of(const void* base, int64_t k_stride, std::initializer_list<int64_t> other_strides, int element) {
    if (k_stride != 1) return Load::AlongRows;
    bool aligned = ((uintptr_t)base & 15) == 0;
    for (int64_t s : other_strides) aligned = aligned && (s * element) % 16 == 0;
    return aligned ? Load::Wide : Load::AlongK;
}

int launch_gemm(const GemmParams& p, cudaStream_t stream) {
    const int element = p.half ? 2 : 4;
    TileArgs args{1, load_of(p.a, p.sa[2], {p.sa[0], p.sa[1]}, element), load_of(p.b, p.sb[1], {p.sb[0], p.sb[2]}, element), p.sc[1] == 1 && p.sc[2] != 1};
    if (p.half) return launch(GemmProblemHalf{p}, p.m, p.n, p.batch, 1, p.k, args, stream);
    const int64_t k_blocks = (p.k + BK - 1) / BK;
    if (p.sb[2] == 1 && cols_fits(p.m, p.n, p.batch, k_blocks)) {
        const bool wide_c = p.sc[2] == 1 && p.n % 4 == 0 && p.sc[0] % 4 == 0 && p.sc[1] % 4 == 0 && ((uintptr_t)p.c & 15) == 0;
        const ColsArgs cols{1, args.load_a, load_of(p.b, p.sb[2], {p.sb[0], p.sb[1]}, 4) == Load::Wide, args.rows_fast, wide_c};
        return launch_cols(GemmProblem{p}, p.m, p.n, p.batch, k_blocks, cols, stream);
    }
    return launch(GemmProblem{p}, p.m, p.n, p.batch, 1, p.k, args, stream);
}

// Matrix multiply with very few output columns (a classifier head, n <= 8): a 64 x 64 tile would leave
// almost every thread idle and walk K serially, so one warp takes one output row instead, its lanes
// stride through K (coalesced when K is the fast axis of both operands) and a shuffle tree sums them.
constexpr int kSkinnyMaxN = 8;

__global__ void __launch_bounds__(256) gemm_skinny_kernel(const __grid_constant__ GemmParams p) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int64_t row_id = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row_id >= p.batch * p.m) return;
    const int64_t b = row_id / p.m, m = row_id - b * p.m;
    const float* a = p.a + b * p.sa[0] + m * p.sa[1];
    const float* w = p.b + b * p.sb[0];
    float acc[kSkinnyMaxN];
#pragma unroll
    for (int n = 0; n < kSkinnyMaxN; n++) acc[n] = 0.f;
    const bool wide = p.sa[2] == 1 && p.sb[1] == 1 && (p.k & 3) == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0 && (p.sb[2] & 3) == 0;
    if (wide) {
        // both operands contiguous along K: 128-bit loads, two per lane in flight for each operand row
        const int64_t k4 = p.k >> 2;
        const float4* a4 = (const float4*)a;
#pragma unroll 2
        for (int64_t k = lane; k < k4; k += 32) {
            const float4 x = __ldg(a4 + k);
#pragma unroll
            for (int n = 0; n < kSkinnyMaxN; n++)
                if (n < p.n) {
                    const float4 y = __ldg((const float4*)(w + n * p.sb[2]) + k);
                    acc[n] = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, acc[n]))));
                }
        }
    } else {
#pragma unroll 4
        for (int64_t k = lane; k < p.k; k += 32) {
            const float x = a[k * p.sa[2]];
#pragma unroll
            for (int n = 0; n < kSkinnyMaxN; n++)
                if (n < p.n) acc[n] = fmaf(x, w[k * p.sb[1] + n * p.sb[2]], acc[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < kSkinnyMaxN; n++)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc[n] += __shfl_xor_sync(0xffffffffu, acc[n], off);
#pragma unroll
    for (int n = 0; n < kSkinnyMaxN; n++) {
        if (n < p.n && lane == n) {
            float v = acc[n];
            if (p.add1) v += p.add1[b * p.s1[0] + m * p.s1[1] + n * p.s1[2]];
            if (p.add2) v += p.add2[b * p.s2[0] + m * p.s2[1] + n * p.s2[2]];
            p.c[b * p.sc[0] + m * p.sc[1] + n * p.sc[2]] = apply_epilogue(v, p.act, p.round_tf32);
        }
    }
}

}  // namespace

int launch_gemm_simt(const GemmParams& p, cudaStream_t stream) {
    if (p.row_softmax == 4) return launch_softmax_matmul(p, stream);
    if (p.half) return launch_gemm(p, stream);
    if (p.n >= 1 && p.n <= kSkinnyMaxN && p.k >= 32 && p.batch * p.m > 0) {
        const int64_t rows = p.batch * p.m;
        launch_pdl(gemm_skinny_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), (size_t)(0), stream, p);
        return (int)cudaGetLastError();
    }
    if (p.m >= 1 && p.m <= kSkinnyMaxN && p.k >= 32 && p.batch * p.n > 0) {
        // few output ROWS (a single token through a linear layer): the same kernel on the transposed problem,
        // C^T = B^T . A^T, one warp per output column
        GemmParams t = p;
        t.a = p.b;
        t.b = p.a;
        t.m = p.n;
        t.n = p.m;
        const int64_t sa[3] = {p.sb[0], p.sb[2], p.sb[1]}, sb[3] = {p.sa[0], p.sa[2], p.sa[1]};
        for (int i = 0; i < 3; i++) {
            t.sa[i] = sa[i];
            t.sb[i] = sb[i];
        }
        std::swap(t.sc[1], t.sc[2]);
        std::swap(t.s1[1], t.s1[2]);
        std::swap(t.s2[1], t.s2[2]);
        const int64_t rows = t.batch * t.m;
        launch_pdl(gemm_skinny_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), (size_t)(0), stream, t);
        return (int)cudaGetLastError();
    }
    return launch_gemm(p, stream);
}

int launch_conv_simt(const ConvParams& p, cudaStream_t stream) {
    TileArgs args{1, load_of(p.in, p.s_in[1], {p.s_in[0], p.s_in[2], p.s_in[3]}, 4), load_of(p.filter, p.s_f[1], {p.s_f[0], p.s_f[2], p.s_f[3]}, 4),
                  p.s_out[1] != 1};
    const int64_t positions = (int64_t)p.n * p.oh * p.ow, k_blocks = (int64_t)p.r * p.s * ((p.c + BK - 1) / BK);
    if (p.s_f[0] == 1 && cols_fits(positions, p.k, 1, k_blocks)) {
        const bool wide_c = p.s_out[1] == 1 && p.k % 4 == 0 && p.s_out[0] % 4 == 0 && p.s_out[2] % 4 == 0 && p.s_out[3] % 4 == 0 && ((uintptr_t)p.out & 15) == 0;
        const ColsArgs cols{1, args.load_a, load_of(p.filter, p.s_f[0], {p.s_f[1], p.s_f[2], p.s_f[3]}, 4) == Load::Wide, args.rows_fast, wide_c};
        return launch_cols(ConvProblem{p}, positions, p.k, 1, k_blocks, cols, stream);
    }
    return launch(ConvProblem{p}, (int64_t)p.n * p.oh * p.ow, p.k, 1, (int64_t)p.r * p.s, p.c, args, stream);
}

}  // namespace kn
