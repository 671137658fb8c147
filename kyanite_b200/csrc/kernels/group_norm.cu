// Group normalisation with its per-channel scale and shift (and SiLU) as one launch: graphs spell it view [N, groups, rest] ->
// layernorm -> view -> multiply -> add (-> times its sigmoid).  Planned node by node that is a layernorm over plain NCHW memory, an
// elementwise step, a transposing copy for the channels-last convolution behind it and, where a channels-last convolution comes
// before it, one more in front: six to eight passes over the tensor and three or four launches.
//
// A group of an image is a cluster of up to eight CTAs, each with a share of it in registers: read once, written once.  A CTA's mean
// and sum of squared deviations (two sweeps over its registers, as the layernorm kernels make them) are merged over the cluster as
// Chan, Golub and LeVeque do for parts of a sample, after one exchange through distributed shared memory (`st.async`, counted by a
// barrier of the receiver: a cluster barrier that releases them takes some 1000 cycles).  Either side may be channels-last; elements
// are numbered in the order of the output, so that stores are whole pieces of its rows.
//
// What bounds it: latency and instructions (tensors of 1 to 16 MB between the convolutions of a denoising step): the loads, the two
// sums, the exchange, then per value a division, a scale, a shift and a SiLU.
// 320 channels of 64 x 64 in 32 groups: 8.9 us in a row of such launches, 640 of 32 x 32 5.7, 960 of 64 x 64 18.7.  Measured against:
// statistics and application as two launches (15.4 us), CTAs of 256 threads with up to 60 values each (18.5: the divisions of a
// thread come one after the other, and a division is a branch), clusters of eight where four hold a group (960 channels 36.6: they
// take two rounds).
#include <cuda_runtime.h>

#include <algorithm>

#include "../kernels.h"
#include "../scalar_ops.h"
#include "launch.cuh"
#include "tc_ptx.cuh"

namespace kn {

namespace {

constexpr int kMaxThreads = 1024;
constexpr int kMaxCluster = 8, kFloats = 8, kMaxFloats = 32;   // values of a thread: as a rule, and where a group is large
constexpr unsigned kFull = 0xffffffffu;

template <int N>
__device__ __forceinline__ float lanes_sum(float x) {
#pragma unroll
    for (int s = N / 2; s > 0; s >>= 1) x += __shfl_xor_sync(kFull, x, s);
    return x;
}
// of a block; in every thread (`shared` is not written by anybody else)
__device__ __forceinline__ float block_sum(float x, float* shared) {
    x = lanes_sum<32>(x);
    const int lane = threadIdx.x & 31;
    if (lane == 0) shared[threadIdx.x >> 5] = x;
    __syncthreads();
    return lanes_sum<32>(lane * 32 < (int)blockDim.x ? shared[lane] : 0.f);
}

template <int V>
__device__ __forceinline__ void load(float (&x)[V], const float* at) {
    if constexpr (V == 4) {
        const float4 v = __ldg((const float4*)at);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    } else if constexpr (V == 2) {
        const float2 v = __ldg((const float2*)at);
        x[0] = v.x, x[1] = v.y;
    } else {
        x[0] = __ldg(at);
    }
}

// V consecutive values of the output: channels of a position (OUT_LAST) or positions of a channel; F values a thread
template <bool IN_LAST, bool OUT_LAST, int V, int F>
__global__ void __launch_bounds__(kMaxThreads) group_norm_kernel(const __grid_constant__ GroupNormParams p) {
    static_assert(IN_LAST == OUT_LAST || V == 1, "pieces lie the same way on both sides");
    constexpr int kItems = F / V;
    __shared__ float sums[kMaxThreads / 32], squares[kMaxThreads / 32];
    __shared__ __align__(8) float2 parts[kMaxCluster];   // mean and sum of squared deviations of each CTA
    __shared__ __align__(8) uint64_t barrier;
    const int cluster = p.cluster;
    const uint32_t arrived = tcp::smem_u32(&barrier);
    if (cluster > 1) {
        if (threadIdx.x == 0) {
            tcp::mbar_init(arrived, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            tcp::mbar_expect_tx(arrived, 8u * (unsigned)cluster);
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (waited for before the first remote store)
    }
    pdl_enter();
    const uint32_t rank = blockIdx.x % (unsigned)cluster;
    const int group = (int)(blockIdx.x / (unsigned)cluster % (unsigned)p.groups);
    const int64_t img = blockIdx.x / (unsigned)cluster / (unsigned)p.groups;
    // pieces are numbered along the output's rows of `row` pieces: channels of a position, or positions of a channel
    const uint32_t row = (uint32_t)(OUT_LAST ? p.group_channels : p.hw) / V;
    const uint32_t pieces = (uint32_t)((int64_t)p.group_channels * p.hw / V), share = (pieces + cluster - 1) / cluster;
    const uint32_t first = min(pieces, rank * share), count = min(pieces, first + share) - first;
    const uint32_t row0 = (first + threadIdx.x) / row, column0 = first + threadIdx.x - row0 * row;
    const uint32_t row_step = blockDim.x / row, column_step = blockDim.x - row_step * row;
    auto advance = [&](uint32_t& r, uint32_t& column) {   // by blockDim.x pieces
        r += row_step, column += column_step;
        if (column >= row) column -= row, r++;
    };
    const int c0 = group * p.group_channels;
    const float* in = p.in + img * p.in_image + (IN_LAST ? c0 : (int64_t)c0 * p.hw);
    float x[kItems][V];
    {
        uint32_t r = row0, column = column0;
#pragma unroll
        for (int i = 0; i < kItems; i++) {
#pragma unroll
            for (int j = 0; j < V; j++) x[i][j] = 0.f;
            if (i * blockDim.x + threadIdx.x < count) {
                const uint32_t channel = OUT_LAST ? column * V : r, position = OUT_LAST ? r : column * V;
                load<V>(x[i], in + (IN_LAST ? (uint64_t)position * (uint32_t)p.in_position + channel : (uint64_t)channel * (uint32_t)p.hw + position));
            }
            advance(r, column);
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kItems; i++)
#pragma unroll
        for (int j = 0; j < V; j++) sum += x[i][j];
    sum = block_sum(sum, sums);
    float mean = count ? sum / (float)(count * V) : 0.f, sq = 0.f;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        if (i * blockDim.x + threadIdx.x >= count) continue;
#pragma unroll
        for (int j = 0; j < V; j++) sq += (x[i][j] - mean) * (x[i][j] - mean);
    }
    sq = block_sum(sq, squares);
    if (cluster > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if ((int)threadIdx.x < cluster)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                         ::"r"(tcp::map_to_cta(tcp::smem_u32(&parts[rank]), threadIdx.x)), "f"(mean), "f"(sq), "r"(tcp::map_to_cta(arrived, threadIdx.x))
                         : "memory");
        const long long start = clock64();
        while (!tcp::mbar_try_wait_cluster(arrived, 0)) {
            if (clock64() - start > tcp::kWaitCycles) {
                atomicMax(p.status, 72u);
                return;
            }
        }
        // lane r (of eight) has part r
        const uint32_t r = threadIdx.x & (kMaxCluster - 1);
        const uint32_t begin = min(pieces, r * share);
        const float n = r < (uint32_t)cluster ? (float)((min(pieces, begin + share) - begin) * V) : 0.f, all = (float)(pieces * V);
        float2 part = make_float2(0.f, 0.f);
        if (n > 0.f) part = parts[r];
        mean = lanes_sum<kMaxCluster>(part.x * (n / all));
        const float delta = part.x - mean;
        sq = lanes_sum<kMaxCluster>(n > 0.f ? part.y + delta * delta * n : 0.f);
    }
    const float denom = sqrtf(sq / (float)(pieces * V) + p.eps), inverse = 1.f / denom;
    const bool normal = divides_by(denom);
    float* out = p.out + img * p.out_image + (OUT_LAST ? c0 : (int64_t)c0 * p.hw);
    const float *scale = p.scale + c0 * p.scale_stride, *shift = p.shift + c0 * p.shift_stride;
    const bool dense = OUT_LAST && p.scale_stride == 1 && p.shift_stride == 1 && ((uintptr_t)scale | (uintptr_t)shift) % (4 * V) == 0;
    uint32_t r = row0, column = column0;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        if (i * blockDim.x + threadIdx.x >= count) break;
        const uint32_t channel = OUT_LAST ? column * V : r, position = OUT_LAST ? r : column * V;
        float y[V], a[V], b[V];
        if (dense) {
            load<V>(a, scale + channel);
            load<V>(b, shift + channel);
        } else {
#pragma unroll
            for (int j = 0; j < V; j++) {
                a[j] = __ldg(scale + (channel + (OUT_LAST ? j : 0)) * p.scale_stride);
                b[j] = __ldg(shift + (channel + (OUT_LAST ? j : 0)) * p.shift_stride);
            }
        }
#pragma unroll
        for (int j = 0; j < V; j++) {
            const float d = x[i][j] - mean;
            y[j] = normal ? divide_by(d, denom, inverse) : d / denom;
            y[j] = __fadd_rn(__fmul_rn(y[j], a[j]), b[j]);
            if (p.silu) y[j] *= 1.0f / (1.0f + expf(-y[j]));
        }
        float* at = out + (OUT_LAST ? (uint64_t)position * (uint32_t)p.out_position + channel : (uint64_t)channel * (uint32_t)p.hw + position);
        if constexpr (V == 4) *(float4*)at = make_float4(y[0], y[1], y[2], y[3]);
        else if constexpr (V == 2) *(float2*)at = make_float2(y[0], y[1]);
        else *at = y[0];
        advance(r, column);
    }
}

template <bool IN_LAST, bool OUT_LAST, int V, int F>
int launch_values(const GroupNormParams& p, int threads, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.images * p.groups * p.cluster));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return (int)cudaLaunchKernelEx(&cfg, group_norm_kernel<IN_LAST, OUT_LAST, V, F>, p);
}

template <bool IN_LAST, bool OUT_LAST, int V>
int launch_pieces(const GroupNormParams& p, cudaStream_t stream) {
    const int64_t pieces = (int64_t)p.group_channels * p.hw / V, share = (pieces + p.cluster - 1) / p.cluster;
    const int threads = (int)std::min<int64_t>(kMaxThreads, (share * V + kFloats * 32 - 1) / (kFloats * 32) * 32);
    const int64_t values = (share + threads - 1) / threads * V;
    if (values <= 4) return launch_values<IN_LAST, OUT_LAST, V, 4>(p, threads, stream);
    if (values <= kFloats) return launch_values<IN_LAST, OUT_LAST, V, kFloats>(p, threads, stream);
    if (values <= 16) return launch_values<IN_LAST, OUT_LAST, V, 16>(p, threads, stream);
    return launch_values<IN_LAST, OUT_LAST, V, kMaxFloats>(p, threads, stream);
}

}  // namespace

// CTAs of a group: as many as give the chip one each, and as its values need; 0 if eight do not hold them.  (120 and not 148: 32 groups, the
// usual number, are 128 CTAs of clusters of four; clusters of eight are two rounds of 960 channels of 64 x 64, 36.6 us instead of 18.7.)
int group_norm_cluster(int64_t groups, int64_t values) {
    for (int c = 1; c <= kMaxCluster; c *= 2)
        if (values <= (int64_t)c * kMaxThreads * kMaxFloats && (groups * c >= 120 || c == kMaxCluster)) return c;
    return 0;
}

int launch_group_norm(const GroupNormParams& p, cudaStream_t stream) {
    if (!p.in_last && p.out_last) return launch_pieces<false, true, 1>(p, stream);
    if (!p.in_last) return launch_pieces<false, false, 4>(p, stream);
    auto whole = [&](int64_t v) {
        return p.group_channels % v == 0 && p.in_position % v == 0 && p.in_image % v == 0 && p.out_position % v == 0 && p.out_image % v == 0 &&
               (uintptr_t)p.in % (4 * v) == 0 && (uintptr_t)p.out % (4 * v) == 0;
    };
    if (whole(4)) return launch_pieces<true, true, 4>(p, stream);
    if (whole(2)) return launch_pieces<true, true, 2>(p, stream);
    return launch_pieces<true, true, 1>(p, stream);
}

}  // namespace kn
