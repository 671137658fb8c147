// Elementwise programs that occur in most networks, compiled instead of interpreted: a residual sum, scale + shift (+ SiLU) of a
// normalisation, the gates of a feed-forward block (SwiGLU, GELU), half of a rotary embedding; f32 or all-f16.
//
// The interpreters of elementwise.cu (scalar_acc_kernel, scalar_h2_kernel) are bound by instructions: decoding a micro-op, parking
// values in shared memory and one load in flight after the other cost them two to four times what these programs need to move
// their operands: half of a rotary embedding of 2048 x 32 x 128 halves 13.4 us there, 7.4 here; scale + shift + SiLU of 1.3 M
// floats 7.5 and 3.7; SwiGLU of 333 x 11008 halves and two sums of 333 x 4096 17.2 us together and 12.3.  Here a program is
// straight-line code: all loads of a thread first (V positions of 16 bytes of each operand, the positions of a block interleaved
// so that a warp reads whole lines), then the arithmetic in registers, then the stores.  The operations and their roundings are
// those of the interpreters, one by one, so the results are the same bit for bit.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../kernels.h"
#include "../scalar_ops.h"
#include "launch.cuh"

namespace kn {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float mul(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ float add(float x, float y) { return __fadd_rn(x, y); }
__device__ __forceinline__ float neg(float x) { return -x; }
__device__ __forceinline__ float sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ __half2 mul(__half2 x, __half2 y) { return __hmul2_rn(x, y); }
__device__ __forceinline__ __half2 add(__half2 x, __half2 y) { return __hadd2_rn(x, y); }
__device__ __forceinline__ __half2 neg(__half2 x) { return __hneg2(x); }
__device__ __forceinline__ __half2 sigmoid(__half2 x) {
    const float2 f = __half22float2(x);
    return __floats2half2_rn(__fdividef(1.0f, 1.0f + __expf(-f.x)), __fdividef(1.0f, 1.0f + __expf(-f.y)));
}

// ---------------------------------------------------------------- the programs
// `ops`: the accumulator program (the planner's allocate_registers) behind the loads, which come in operand order, and in front of
// the store; 255 is the accumulator.  `eval`: the same as code; `c` holds the constants of the operations of kind 5 in order.
struct MicroOp {
    uint8_t kind, op, a, b, slot;   // (b: of kind 2)
};
constexpr uint8_t kAcc = 255;
constexpr uint8_t kAdd = (uint8_t)BinaryOp::Add, kMul = (uint8_t)BinaryOp::Mul;
constexpr int kMaxOps = 8, kMaxLoads = 4;

struct Sum {   // x + y
    static constexpr int kLoads = 2, kParked = 1, kOps = 1;
    static constexpr MicroOp ops[kOps] = {{2, kAdd, 0, kAcc, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) { return add(x[0], x[1]); }
};
struct Affine {   // x * scale + shift
    static constexpr int kLoads = 3, kParked = 3, kOps = 2;
    static constexpr MicroOp ops[kOps] = {{2, kMul, 0, 1, kAcc}, {2, kAdd, kAcc, 2, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) { return add(mul(x[0], x[1]), x[2]); }
};
struct AffineSilu {   // y * sigmoid(y), y = x * scale + shift
    static constexpr int kLoads = 3, kParked = 3, kOps = 4;
    static constexpr MicroOp ops[kOps] = {
        {2, kMul, 0, 1, kAcc}, {2, kAdd, kAcc, 2, 2}, {1, (uint8_t)UnaryOp::Sigmoid, kAcc, 0, kAcc}, {2, kMul, 2, kAcc, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) {
        const X y = add(mul(x[0], x[1]), x[2]);
        return mul(y, sigmoid(y));
    }
};
struct SwiGlu {   // gate * sigmoid(gate) * x
    static constexpr int kLoads = 2, kParked = 2, kOps = 3;
    static constexpr MicroOp ops[kOps] = {{1, (uint8_t)UnaryOp::Sigmoid, 0, 0, kAcc}, {2, kMul, 0, kAcc, kAcc}, {2, kMul, kAcc, 1, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) { return mul(mul(x[0], sigmoid(x[0])), x[1]); }
};
struct GeluGate {   // x * (gate * c0) * (erf(gate * c1) + c2): f32 only
    static constexpr int kLoads = 2, kParked = 2, kOps = 6;
    static constexpr MicroOp ops[kOps] = {{5, kMul, kAcc, 0, 2}, {5, kMul, 1, 0, kAcc}, {1, (uint8_t)UnaryOp::Erf, kAcc, 0, kAcc},
                                          {5, kAdd, kAcc, 0, kAcc}, {2, kMul, 2, kAcc, kAcc}, {2, kMul, 0, kAcc, kAcc}};
    static __device__ float eval(const float (&x)[kLoads], const float* c) {
        return mul(x[0], mul(mul(x[1], c[0]), add(erff(mul(x[1], c[1])), c[2])));
    }
};
struct RotaryFirst {   // x * cos + (-y) * sin
    static constexpr int kLoads = 4, kParked = 4, kOps = 4;
    static constexpr MicroOp ops[kOps] = {{2, kMul, 0, 1, 1}, {1, (uint8_t)UnaryOp::Neg, 2, 0, kAcc}, {2, kMul, kAcc, 3, kAcc}, {2, kAdd, 1, kAcc, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) { return add(mul(x[0], x[1]), mul(neg(x[2]), x[3])); }
};
struct RotarySecond {   // y * cos + x * sin
    static constexpr int kLoads = 4, kParked = 4, kOps = 3;
    static constexpr MicroOp ops[kOps] = {{2, kMul, 0, 1, 1}, {2, kMul, 2, 3, kAcc}, {2, kAdd, 1, kAcc, kAcc}};
    template <class X> static __device__ X eval(const X (&x)[kLoads], const float*) { return add(mul(x[0], x[1]), mul(x[2], x[3])); }
};

struct FixedParams {
    uint32_t total;                 // positions of 16 bytes
    int32_t rank;
    uint32_t dims[DEV_MAX_RANK];    // the innermost one in positions
    const void* ptr[kMaxLoads + 1];
    uint32_t strides[kMaxLoads + 1][DEV_MAX_RANK];   // in elements; of the innermost axis: per position, 0 = broadcast
    float imm[4];
};

template <class P, bool HALF>
__device__ __forceinline__ uint4 evaluate(const uint4 (&x)[P::kLoads], const float* c) {
    uint4 r;
    if constexpr (HALF) {
        __half2 in[4][P::kLoads];
#pragma unroll
        for (int o = 0; o < P::kLoads; o++)
#pragma unroll
            for (int i = 0; i < 4; i++) in[i][o] = ((const __half2*)&x[o])[i];
#pragma unroll
        for (int i = 0; i < 4; i++) ((__half2*)&r)[i] = P::eval(in[i], c);
    } else {
        float in[4][P::kLoads];
#pragma unroll
        for (int o = 0; o < P::kLoads; o++)
#pragma unroll
            for (int i = 0; i < 4; i++) in[i][o] = ((const float*)&x[o])[i];
#pragma unroll
        for (int i = 0; i < 4; i++) ((float*)&r)[i] = P::eval(in[i], c);
    }
    return r;
}

template <class P, bool HALF, int V, bool RANK1>
__global__ void __launch_bounds__(kThreads) scalar_fixed_kernel(const __grid_constant__ FixedParams p) {
    constexpr int kOperands = P::kLoads + 1;
    using T = typename std::conditional<HALF, __half, float>::type;
    pdl_enter();
    uint4 x[V][P::kLoads];
    uint32_t to[V];
    const uint32_t first = blockIdx.x * (kThreads * V) + threadIdx.x;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const uint32_t at = first + v * kThreads;
        if (at >= p.total) break;
        uint32_t off[kOperands];
        if (RANK1) {
#pragma unroll
            for (int o = 0; o < kOperands; o++) off[o] = at * p.strides[o][0];
        } else {
#pragma unroll
            for (int o = 0; o < kOperands; o++) off[o] = 0;
            uint32_t rem = at;
            for (int d = p.rank - 1; d >= 0; d--) {
                const uint32_t q = d > 0 ? rem / p.dims[d] : 0u, i = rem - q * p.dims[d];
                rem = q;
#pragma unroll
                for (int o = 0; o < kOperands; o++) off[o] += i * p.strides[o][d];
            }
        }
        to[v] = off[P::kLoads];
#pragma unroll
        for (int o = 0; o < P::kLoads; o++) {
            const T* src = (const T*)p.ptr[o] + off[o];
            if (p.strides[o][RANK1 ? 0 : p.rank - 1] != 0) {
                x[v][o] = __ldg((const uint4*)src);
            } else if (HALF) {
                const uint32_t w = (uint32_t)__ldg((const unsigned short*)src) * 0x00010001u;
                x[v][o] = make_uint4(w, w, w, w);
            } else {
                const uint32_t w = __ldg((const uint32_t*)src);
                x[v][o] = make_uint4(w, w, w, w);
            }
        }
    }
#pragma unroll
    for (int v = 0; v < V; v++) {
        if (first + v * kThreads >= p.total) break;
        *(uint4*)((T*)const_cast<void*>(p.ptr[P::kLoads]) + to[v]) = evaluate<P, HALF>(x[v], p.imm);
    }
}

// The program is `P`, in f32 or f16
template <class P>
bool matches(const ScalarParams& p, DType type) {
    if (p.n_loads != P::kLoads || p.n_operands != P::kLoads + 1 || p.n_stores != 1 || p.n_micro != P::kLoads + P::kOps + 1) return false;
    for (int o = 0; o < P::kLoads; o++) {
        const ScalarInstr& m = p.micro[o];
        if (m.kind != 3 || m.a != o || (m.pad & 0xFF) != (o < P::kParked ? o : kAcc)) return false;
    }
    for (int i = 0; i < P::kOps; i++) {
        const ScalarInstr& m = p.micro[P::kLoads + i];
        const MicroOp& want = P::ops[i];
        if (m.kind != want.kind || m.op != want.op || m.a != want.a || (m.kind == 2 && m.b != want.b) || (m.pad & 0xFF) != want.slot) return false;
        if (m.dtype != (uint8_t)type) return false;
    }
    const ScalarInstr& store = p.micro[p.n_micro - 1];
    return store.kind == 4 && store.a == kAcc && store.b == P::kLoads;
}

template <class P, bool HALF, int V>
int launch_fixed(const FixedParams& f, cudaStream_t stream) {
    const dim3 grid((f.total + kThreads * V - 1) / (kThreads * V));
    if (f.rank == 1) launch_pdl(scalar_fixed_kernel<P, HALF, V, true>, grid, dim3(kThreads), (size_t)0, stream, f);
    else launch_pdl(scalar_fixed_kernel<P, HALF, V, false>, grid, dim3(kThreads), (size_t)0, stream, f);
    return (int)cudaGetLastError();
}

template <class P, bool HALF>
int launch_program(const ScalarParams& p, cudaStream_t stream) {
    constexpr int64_t kElements = HALF ? 8 : 4;
    FixedParams f = {};
    f.total = (uint32_t)(p.total / kElements);
    f.rank = p.rank;
    const int last = p.rank - 1;
    for (int d = 0; d < p.rank; d++) f.dims[d] = (uint32_t)(d == last ? p.dims[d] / kElements : p.dims[d]);
    for (int o = 0; o <= P::kLoads; o++) {
        f.ptr[o] = p.ptr[o];
        for (int d = 0; d < p.rank; d++) f.strides[o][d] = (uint32_t)(p.strides[o][d] * (d == last ? kElements : 1));
    }
    int n = 0;
    for (int i = 0; i < P::kOps; i++)
        if (P::ops[i].kind == 5) f.imm[n++] = bits_to_f32(p.micro[P::kLoads + i].imm);
    // One position a thread, two of programs of two loads from a million positions on. Sum in f32, 5.2 M elements: 6.4 us with
    // one, 5.2 with two; 2.6 M 4.5 with either. SwiGLU 5.2 M 6.7 and 6.4, 2.6 M 4.0 and 4.3. Scale + shift + SiLU 5.2 M 9.8 and
    // 10.7, 1.3 M 3.7 and 5.0. (Four were no faster anywhere.)
    if (P::kLoads <= 2 && f.total >= 1000000u) return launch_fixed<P, HALF, 2>(f, stream);
    return launch_fixed<P, HALF, 1>(f, stream);
}

template <bool HALF>
int launch_one(const ScalarParams& p, cudaStream_t stream) {
    switch (p.fixed) {
        case 1: return launch_program<Sum, HALF>(p, stream);
        case 2: return launch_program<Affine, HALF>(p, stream);
        case 3: return launch_program<AffineSilu, HALF>(p, stream);
        case 4: return launch_program<SwiGlu, HALF>(p, stream);
        case 5: return launch_program<RotaryFirst, HALF>(p, stream);
        case 6: return launch_program<RotarySecond, HALF>(p, stream);
        default: break;
    }
    if constexpr (!HALF)
        if (p.fixed == 7) return launch_program<GeluGate, HALF>(p, stream);
    return (int)cudaErrorInvalidValue;
}

}  // namespace

int scalar_fixed_program(const ScalarParams& p, bool half) {
    const DType type = half ? DType::F16 : DType::F32;
    if (matches<Sum>(p, type)) return 1;
    if (matches<Affine>(p, type)) return 2;
    if (matches<AffineSilu>(p, type)) return 3;
    if (matches<SwiGlu>(p, type)) return 4;
    if (matches<RotaryFirst>(p, type)) return 5;
    if (matches<RotarySecond>(p, type)) return 6;
    if (!half && matches<GeluGate>(p, type)) return 7;
    return 0;
}

int launch_scalar_fixed(const ScalarParams& p, cudaStream_t stream) {
    return p.vec4 == 5 ? launch_one<true>(p, stream) : launch_one<false>(p, stream);
}

}  // namespace kn
