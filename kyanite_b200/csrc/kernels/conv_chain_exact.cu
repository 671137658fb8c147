// A run of 3x3 stride-1 same-padding convolutions in exact f32 as ONE kernel (sm_100a): a cluster of CTAs per image.
//
// The exact counterpart of conv_chain.cu for batches of at most one cluster per image on the chip.  One launch per layer
// (contract_cols_kernel) pays for every layer the launch, the pipeline's fill, a round of tiles that does not divide by the SMs and
// the activations' way through L2; here an image's activations lie in the shared memory of every CTA of its cluster, each CTA
// computes its share of the output channels for all positions, and sends them to the others (`st.async`, which counts its bytes on
// the receiver's barrier: no release at cluster scope, which costs 1000 cycles).
//
// A thread computes one image row (8 positions) x 8 channels over its group's share of the input channels: per input channel and
// filter row it reads the row's ten values once for all three taps, 4 reads next to 6 of weights for 96 packed multiply-adds
// (fma.rn.f32x2 over channel pairs).  The groups' partial sums meet in shared memory, four positions of a channel at a time.
// Weights stream through a ring by bulk copies, prefetched across layers.
//
// What bounds it: instruction issue.  An input channel is 288 packed multiply-adds a thread, which issue every other cycle, and some
// 120 reads and moves beside them: 780 cycles for 576 (plain multiply-adds: 940).  The rest of a layer is partial sums, the wait for
// the slowest CTA of the cluster and remote stores at 16 bytes a cycle: some 7 000 of 58 000 cycles at two CTAs an image, and at
// sixteen, whose arithmetic is 3 000, five sixths of them.  64 boards of 8 x 8, 128 channels: 36.5 us a layer launched one by one,
// 29.7 here (0.55 of the multiply-add rate).
//
// Every wait is bounded; on expiry the executor's status word is raised and all roles leave.
#include <cuda_runtime.h>

#include <algorithm>
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

constexpr int kWorkers = 256;
constexpr int kPitch = 12;       // floats of an image row in shared memory: x = 0 .. w - 1, then zeros (x = -1 is the row before's last)
constexpr int W = 8;             // positions of a row that a thread computes
constexpr int kQuads = W / 4;    // groups of four positions
constexpr int kSums = 8 * kQuads;            // partial sums of a thread, in float4
// Products that a thread sums one behind the other, about: the sums of such segments of its input channels are summed by themselves, and
// so are four groups' at a time.  With one sum over all of a thread's products chains were up to twice as far from 64 bits as
// the layers launched one by one (nine layers of 128 channels: 130 boards 1.98 times, 46 1.44, 25 1.17); now 0.70 to 1.00 times.  A
// segment's end costs 0.5 to 0.9 us a layer and moves 64 boards from 29.0 to 29.7 us a layer.  (At 72 products 64 boards took
// 30.7; sums kept in tensor memory instead of shared memory no less.)
constexpr int kSegment = 96;

struct ExactKernelParams {
    const float* in;
    float* out;
    const float* bias;
    const float* weights;
    int64_t s_in[4], s_out[4];
    int32_t c_in, k, h, w;
    int32_t n_layers, cluster, cols, k_groups, items;   // cols: output channels of a CTA; items: (image row, 8 of them)
    int32_t chunk, slots, channels;      // input channels of a weight chunk; ring slots; input channels that shared memory holds
    int32_t segment;                     // chunks that are summed by themselves, or 0: all of them
    int32_t act_floats;                  // of a channel: (h + 2) * kPitch
    uint8_t flags[kMaxChainLayers];
    uint8_t chunks[kMaxChainLayers];     // weight chunks of the layer
    uint32_t* status;
};

__device__ __forceinline__ void store_async(uint32_t addr, uint32_t bar, float4 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}

// U: results of a thread, in groups of four (at most).  SEGMENTED: a layer's input channels are more than one segment
template <int U, bool SEGMENTED>
__global__ void __launch_bounds__(kWorkers, 1)
conv_chain_exact_kernel(const __grid_constant__ ExactKernelParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    const int act_bytes = (p.channels * p.act_floats + kPitch) * 4;       // (a row in front: x = -1 of the first)
    float* const act = (float*)smem + kPitch;
    const int partial_at = (act_bytes + 15) & ~15;
    float4* const partial = (float4*)(smem + partial_at);
    const int ring_at = (partial_at + kWorkers * kSums * 16 + 127) & ~127;
    const uint32_t chunk_bytes = (uint32_t)(p.chunk * 9 * p.cols * 4);
    const uint32_t bars = base + (uint32_t)ring_at + (uint32_t)p.slots * chunk_bytes;
    const uint32_t full_bar = bars, empty_bar = full_bar + 8u * p.slots, act_full = empty_bar + 8u * p.slots, ready = act_full + 8u;
    volatile int* abandon = (volatile int*)(smem + (ready + 8u - base));

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int64_t img = blockIdx.x / (unsigned)p.cluster;
    if (tid == 0) {
        for (int s = 0; s < p.slots; s++) {
            mbar_init(full_bar + 8u * s, 1);
            mbar_init(empty_bar + 8u * s, kWorkers / 32);
        }
        mbar_init(act_full, 1);
        mbar_init(ready, (uint32_t)p.cluster);
        *abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < act_bytes / 4; i += kWorkers) ((float*)smem)[i] = 0.f;
    __syncthreads();
    if (p.cluster > 1) cluster_sync_all();   // the peers' barriers are initialised before anything is sent to them

    // Weights: thread 0 keeps the ring full, two chunks behind the one it consumes.  They are a constant of the plan: nothing
    // here waits for the previous kernel.
    int load_layer = 0, load_chunk = 0, load_slot = 0, load_round = 0;
    const char* load_from = (const char*)p.weights + (size_t)rank * p.chunks[0] * chunk_bytes;
    auto load_next = [&]() -> bool {
        if (load_layer == p.n_layers) return true;
        if (load_round > 0 && !mbar_wait(empty_bar + 8u * load_slot, (uint32_t)((load_round & 1) ^ 1), abandon, p.status, 61)) return false;
        mbar_expect_tx(full_bar + 8u * load_slot, chunk_bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(base + (uint32_t)ring_at + (uint32_t)load_slot * chunk_bytes), "l"(load_from), "r"(chunk_bytes), "r"(full_bar + 8u * load_slot)
                     : "memory");
        load_from += chunk_bytes;
        if (++load_slot == p.slots) load_slot = 0, load_round++;
        if (++load_chunk == p.chunks[load_layer]) {
            load_from += (size_t)(p.cluster - 1 - (int)rank) * load_chunk * chunk_bytes;   // the other CTAs' shares
            load_chunk = 0;
            if (++load_layer < p.n_layers) load_from += (size_t)rank * p.chunks[load_layer] * chunk_bytes;
        }
        return true;
    };
    if (tid == 0)
        for (int i = 0; i < p.slots - 2; i++) load_next();
    {
        const int items = p.items;
        const int group = tid / items, item = tid - group * items;      // (threads past the last group: no input channels)
        const int row = item % p.h, cg = item / p.h;
        const bool works = group < p.k_groups;
        const int per_group = p.chunk / p.k_groups;                     // input channels of a group in a chunk
        // my results: unit u = tid + 256 i is (item, channel, quad of positions)
        const int n_units = items * kSums;
        float4 held[U];
#pragma unroll
        for (int i = 0; i < U; i++) held[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        struct Unit { int item, channel, quad, row; };                  // channel: of all
        auto unit_at = [&](int u) {
            Unit r;
            const int i = u / items;
            r.item = u - i * items;
            r.quad = i % kQuads;
            r.row = r.item % p.h;
            r.channel = (int)rank * p.cols + (r.item / p.h) * 8 + i / kQuads;
            return r;
        };
        // (worked out once: divisions cost as much as everything else that a layer does for a result)
        int at[U], from[U];             // where it goes in `act`, where its first partial sum is
        int channel[U];
        uint32_t edge = 0;              // bit 4 i + x: position x of unit i is past the image
#pragma unroll
        for (int i = 0; i < U; i++) {
            const int t = tid + i * kWorkers;
            const Unit u = unit_at(t < n_units ? t : 0);
            at[i] = u.channel * p.act_floats + (u.row + 1) * kPitch + u.quad * 4;
            from[i] = ((u.channel & 7) * kQuads + u.quad) * kWorkers + u.item;
            channel[i] = u.channel;
#pragma unroll
            for (int x = 0; x < 4; x++) edge |= (uint32_t)(u.quad * 4 + x >= p.w) << (4 * i + x);
        }
        auto has_unit = [&](int i) { return tid + i * kWorkers < n_units; };
        auto sync_workers = [&] { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); };
        // the input
        asm volatile("griddepcontrol.wait;" ::: "memory");
        {
            const int positions = p.h * p.w;
            for (int e = tid; e < p.c_in * positions; e += kWorkers) {
                const bool last = p.s_in[1] == 1;    // (channels contiguous: consecutive threads take consecutive channels)
                const int c = last ? e % p.c_in : e / positions, at = last ? e / p.c_in : e - c * positions;
                const int y = at / p.w, x = at - y * p.w;
                act[c * p.act_floats + (y + 1) * kPitch + x] = p.in[img * p.s_in[0] + c * p.s_in[1] + y * p.s_in[2] + x * p.s_in[3]];
            }
            sync_workers();
            if (p.c_in == p.k) {
#pragma unroll
                for (int i = 0; i < U; i++) {
                    if (has_unit(i)) held[i] = *(const float4*)(act + at[i]);
                }
            }
        }
        // the ten values around a row's positions (x = -1 is the row before's last element, a zero)
        auto load_row = [](float (&a)[W + 2], const float* from) {
            a[0] = from[-1];
#pragma unroll
            for (int q = 0; q < W / 4; q++) {
                const float4 t = *(const float4*)(from + 4 * q);
                a[1 + 4 * q] = t.x, a[2 + 4 * q] = t.y, a[3 + 4 * q] = t.z, a[4 + 4 * q] = t.w;
            }
            a[W + 1] = from[W];
        };
        int slot = 0, round = 0;
        bool ok = true;
        for (int l = 0; l < p.n_layers; l++) {
            const uint32_t flags = p.flags[l];
            const bool last = l == p.n_layers - 1;
            float b[U];
#pragma unroll
            for (int i = 0; i < U; i++) b[i] = p.bias[l * 128 + channel[i]];
            if (l > 0) ok = mbar_wait_cluster(act_full, (uint32_t)((l - 1) & 1), abandon, p.status, 62);
            const float* a_at = act + (works ? group * per_group : 0) * p.act_floats + row * kPitch;
            const int chunks = p.chunks[l];
            ok = __all_sync(0xffffffffu, ok);   // (the lanes of a warp waited one by one, and vote in the loop)
            if (last && tid == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            int c = 0;
            do {   // (a segment)
                const int from_c = c, to = SEGMENTED ? min(chunks, c + p.segment) : chunks;
                float2 acc[W][4];
#pragma unroll
                for (int x = 0; x < W; x++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[x][j] = make_float2(0.f, 0.f);
                for (; c < to && ok; c++, a_at += p.chunk * p.act_floats) {
                    if (tid == 0) ok = load_next();
                    ok = ok && mbar_wait(full_bar + 8u * slot, (uint32_t)(round & 1), abandon, p.status, 63);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (works) {
                        // Loads run one step ahead of their use: the weights of the next tap, the values of the next filter row
                        const float* a_row = a_at;
                        const float* w_at = (const float*)(smem + ring_at + slot * (int)chunk_bytes) + group * per_group * 9 * p.cols + cg * 8;
                        float a[W + 2];
                        float4 w0 = *(const float4*)w_at, w1 = *(const float4*)(w_at + 4);
                        load_row(a, a_row);
#pragma unroll 1
                        for (int left = per_group; left > 0; left--) {
                            const float* a_next = left > 1 ? a_row + p.act_floats : a_row;
#pragma unroll
                            for (int dy = 0; dy < 3; dy++) {
                                float b[W + 2];
                                load_row(b, dy < 2 ? a_row + (dy + 1) * kPitch : a_next);
#pragma unroll
                                for (int dx = 0; dx < 3; dx++) {
                                    if (dy * 3 + dx < 8 || left > 1) w_at += p.cols;   // (the chunk's last tap: read once more)
                                    const float4 n0 = *(const float4*)w_at, n1 = *(const float4*)(w_at + 4);
                                    const float2 w[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y), make_float2(w1.z, w1.w)};
#pragma unroll
                                    for (int j = 0; j < 4; j++)
#pragma unroll
                                        for (int x = 0; x < W; x++) acc[x][j] = fma_pair(make_float2(a[x + dx], a[x + dx]), w[j], acc[x][j]);
                                    w0 = n0, w1 = n1;
                                }
#pragma unroll
                                for (int x = 0; x < W + 2; x++) a[x] = b[x];
                            }
                            a_row = a_next;
                        }
                    }
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar + 8u * slot) : "memory");
                    if (++slot == p.slots) { slot = 0; round++; }
                }
                // partial sums, [quad of a channel][thread]
                if (!SEGMENTED || from_c == 0) {
#pragma unroll
                    for (int ch = 0; ch < 8; ch++)
#pragma unroll
                        for (int q = 0; q < kQuads; q++) {
                            float v[4];
#pragma unroll
                            for (int x = 0; x < 4; x++) v[x] = ch & 1 ? acc[4 * q + x][ch / 2].y : acc[4 * q + x][ch / 2].x;
                            partial[(ch * kQuads + q) * kWorkers + tid] = make_float4(v[0], v[1], v[2], v[3]);
                        }
                } else {
#pragma unroll
                    for (int ch = 0; ch < 8; ch++)
#pragma unroll
                        for (int q = 0; q < kQuads; q++) {
                            float v[4];
#pragma unroll
                            for (int x = 0; x < 4; x++) v[x] = ch & 1 ? acc[4 * q + x][ch / 2].y : acc[4 * q + x][ch / 2].x;
                            float4& at = partial[(ch * kQuads + q) * kWorkers + tid];
                            const float4 t = at;
                            at = make_float4(t.x + v[0], t.y + v[1], t.z + v[2], t.w + v[3]);
                        }
                }
            } while (SEGMENTED && c < chunks && ok);
            if (tid == 0 && !last) mbar_expect_tx(act_full, (uint32_t)(n_units * p.cluster) * 16u);   // the next layer's input
            {   // (the workers agree on going on: none may be left waiting in a barrier)
                uint32_t all;
                asm volatile(
                    "{\n\t.reg .pred p, q;\n\t"
                    "setp.ne.u32 p, %1, 0;\n\t"
                    "bar.red.and.pred q, 1, 256, p;\n\t"
                    "selp.u32 %0, 1, 0, q;\n\t}"
                    : "=r"(all)
                    : "r"((uint32_t)ok)
                    : "memory");
                if (!all) break;
            }
            if (l == 0 && p.c_in > p.k && p.channels > p.k) {
                // an input wider than the trunk: the channels that whole chunks add to the next layers are none of it (zero weights
                // make NaN of an infinity)
                for (int i = p.k * p.act_floats + tid; i < p.channels * p.act_floats; i += kWorkers) act[i] = 0.f;
                sync_workers();
            }
            // this CTA has read its input: the cluster may write the next layer's over it
            if (!last && tid < p.cluster) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(ready, (uint32_t)tid)) : "memory");
            float4 y[U];
#pragma unroll
            for (int i = 0; i < U; i++) {
                if (!has_unit(i)) continue;
                float4 s = partial[from[i]];
                int g = 1;
#pragma unroll 2
                for (; g + 4 <= p.k_groups; g += 4) {
                    float4 t[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) t[q] = partial[from[i] + (g + q) * items];
                    s.x += (t[0].x + t[1].x) + (t[2].x + t[3].x), s.y += (t[0].y + t[1].y) + (t[2].y + t[3].y);
                    s.z += (t[0].z + t[1].z) + (t[2].z + t[3].z), s.w += (t[0].w + t[1].w) + (t[2].w + t[3].w);
                }
#pragma unroll 1
                for (; g < p.k_groups; g++) {
                    const float4 t = partial[from[i] + g * items];
                    s.x += t.x, s.y += t.y, s.z += t.z, s.w += t.w;
                }
                s.x += b[i], s.y += b[i], s.z += b[i], s.w += b[i];
                if (flags & kChainFlagAddHeld) s.x += held[i].x, s.y += held[i].y, s.z += held[i].z, s.w += held[i].w;
                if (flags & kChainFlagRelu) s.x = fmaxf(s.x, 0.f), s.y = fmaxf(s.y, 0.f), s.z = fmaxf(s.z, 0.f), s.w = fmaxf(s.w, 0.f);
                if (flags & kChainFlagHold) held[i] = s;
                // (columns past the image are the zeros around it)
                if (edge >> (4 * i) & 1) s.x = 0.f;
                if (edge >> (4 * i) & 2) s.y = 0.f;
                if (edge >> (4 * i) & 4) s.z = 0.f;
                if (edge >> (4 * i) & 8) s.w = 0.f;
                y[i] = s;
            }
            if (flags & kChainFlagStore) {
#pragma unroll
                for (int i = 0; i < U; i++) {
                    if (!has_unit(i)) continue;
                    const Unit u = unit_at(tid + i * kWorkers);
                    float* o = p.out + img * p.s_out[0] + u.channel * p.s_out[1] + u.row * p.s_out[2] + u.quad * 4 * p.s_out[3];
                    const float v[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
#pragma unroll
                    for (int x = 0; x < 4; x++)
                        if (!(edge >> (4 * i + x) & 1)) o[x * p.s_out[3]] = v[x];
                }
            }
            if (last) break;
            ok = mbar_wait_cluster(ready, (uint32_t)(l & 1), abandon, p.status, 64);
            if (ok) {
                for (uint32_t r = 0; r < (uint32_t)p.cluster; r++) {
                    const uint32_t to = map_to_cta(smem_u32(act), r), bar = map_to_cta(act_full, r);
#pragma unroll
                    for (int i = 0; i < U; i++)
                        if (has_unit(i)) store_async(to + (uint32_t)at[i] * 4u, bar, y[i]);
                }
            }
        }
    }
    __syncthreads();
    if (p.cluster > 1) cluster_sync_all();   // nobody leaves while it may still be written to
}

struct ExactLaunch {
    ExactKernelParams p;
    unsigned grid;
    int smem_bytes;
    int units;
};

}  // namespace

// Clusters of 16, 8, 4, 2 and 1 CTAs that the chip holds at once, one CTA per SM (cudaOccupancyMaxActiveClusters).
static const int kClusterSizes[5] = {16, 8, 4, 2, 1}, kClustersFit[5] = {7, 15, 33, 74, 148};

// The layers take the same time however many of the clusters of a round there are, so the rule looks at how full the round is:
// us a layer, launched one by one -> as a chain, 8 x 8 boards (13 layers, the first of 21 channels). 128 channels, 6 boards (16 CTAs
// each) 12.2 -> 7.8, 5 7.9 -> 7.8; 12 (8) 19.1 -> 11.0, 11 10.7 -> 11.0; 24 (4) 23.9 -> 15.3, 20 13.8 -> 15.3; 45 (2) 31.6 -> 26.6, 40
// 23.0 -> 26.6; 120 (1) 68.4 -> 53.0, 112 64.0 -> 53.1, 110 49.0 -> 53.1. 64 channels: faster at every size, 0.42 to 0.87 of the time,
// at 0.46 and more of a round or with eight CTAs an image. (Two batches of 22 boards at once: two chains of 0.67 of a round do not run
// side by side, 1038 us against 1008 launched one by one, which is why 0.6 to 0.7 of a round, where a chain alone gains 0 to 6%, is
// left out.)
// Other heights: five boards of 16 x 8 take 1.4 times as long as a chain, six 0.80, 48 of 5 x 8 1.04, 60 0.85. Rows of 7 leave an eighth
// of a thread's work unused: 140 boards of 7 x 7 1.05, 146 0.81.
bool conv_chain_exact_geometry(int h, int w, int64_t n_img, int c_in, int k, ChainExactGeometry* out) {
    if (w < 7 || w > W || h < 4 || h > 16 || n_img < 1 || c_in < 1 || c_in > 128 || k < 32 || k > 128 || k % 8 != 0) return false;
    ChainExactGeometry g{};
    for (int i = 0; i < 5; i++) {
        const int cluster = kClusterSizes[i];
        if (k % (8 * cluster) != 0 || n_img > kClustersFit[i]) continue;
        const double used = (double)(n_img * w) / (W * kClustersFit[i]);
        const double least_used = cluster == 16 ? (h > 8 ? 0.8 : 0.7) : cluster == 8 ? 0.78 : cluster == 4 ? 0.7 : cluster == 2 ? (h == 8 ? 0.6 : 0.7) : 0.72;
        if (k > 64 ? used < least_used : cluster < 8 && used < 0.45) return false;
        if (k > 64 && cluster == 1 && n_img * h * w <= 7104) return false;   // (222 tiles of 64 x 64: three CTAs of half a tile's K an SM)
        g.cluster = cluster;
        g.cols = k / cluster;
        g.items = h * g.cols / 8;
        if (g.items > kWorkers) continue;
        g.units = (g.items * kSums + kWorkers - 1) / kWorkers;
        if (g.units > 8) continue;
        // as few groups as give each its least number of input channels; chunks of at most about 18 KB of whole channels of every
        // group, the larger the better where no more channels are padded
        const int share = (k + kWorkers / g.items - 1) / (kWorkers / g.items);
        g.k_groups = (k + share - 1) / share;
        const int channel_bytes = 9 * g.cols * 4;
        g.act_floats = (h + 2) * kPitch;
        int least = 0;
        for (int per_group = std::max(1, std::min(share, 18 * 1024 / (g.k_groups * channel_bytes))); per_group >= 1; per_group--) {
            const int chunk = g.k_groups * per_group, padded = (k + chunk - 1) / chunk * chunk;
            const int channels = std::max(padded, (c_in + chunk - 1) / chunk * chunk);
            const int fixed = (channels * g.act_floats + kPitch) * 4 + 16 + kWorkers * kSums * 16 + 128 + 16 * 8 + 64;
            const int slots = std::min(8, (227 * 1024 - fixed) / (chunk * channel_bytes));
            if (slots < 4 || (least != 0 && padded >= least)) continue;
            least = padded;
            g.chunk = chunk;
            g.channels = channels;
            g.slots = slots;
            g.smem_bytes = fixed + slots * chunk * channel_bytes;
        }
        if (least == 0) continue;
        if (out) *out = g;
        return true;
    }
    return false;
}

std::shared_ptr<void> chain_exact_prepare(const ConvChainParams& c, uint32_t* status_word) {
    auto l = std::make_shared<ExactLaunch>();
    ExactKernelParams& p = l->p;
    memset(&p, 0, sizeof(p));
    ChainExactGeometry g;
    KN_CHECK(c.n_heads == 0 && conv_chain_exact_geometry(c.h, c.w, c.n, c.c_in, c.k, &g), KN_ERR_INTERNAL, "exact convolution chain does not fit");
    p.in = c.in;
    p.out = c.out;
    p.bias = c.bias;
    p.weights = c.tiles;
    for (int i = 0; i < 4; i++) {
        p.s_in[i] = c.s_in[i];
        p.s_out[i] = c.s_out[i];
    }
    p.c_in = c.c_in;
    p.k = c.k;
    p.h = c.h;
    p.w = c.w;
    p.n_layers = c.n_layers;
    p.cluster = g.cluster;
    p.cols = g.cols;
    p.k_groups = g.k_groups;
    p.items = g.items;
    p.chunk = g.chunk;
    const int chunks = (c.k + g.chunk - 1) / g.chunk, products = 9 * g.chunk / g.k_groups;   // of a thread in a chunk
    const int segments = std::max((chunks * products + kSegment - 1) / kSegment, chunks * products > kSegment / 2 ? 2 : 1);
    p.segment = segments > 1 ? (chunks + segments - 1) / segments : 0;
    p.slots = g.slots;
    p.channels = g.channels;
    p.act_floats = g.act_floats;
    for (int i = 0; i < c.n_layers; i++) {
        p.flags[i] = c.flags[i];
        p.chunks[i] = (uint8_t)(((i == 0 ? c.c_in : c.k) + g.chunk - 1) / g.chunk);
    }
    p.status = status_word;
    l->grid = (unsigned)(c.n * g.cluster);
    l->smem_bytes = g.smem_bytes;
    l->units = g.units;
    return l;
}

int chain_exact_launch(const void* launch, cudaStream_t stream) {
    const ExactLaunch& l = *(const ExactLaunch*)launch;
    static std::mutex mu;
    static bool done[4][64] = {};
    const bool segmented = l.p.segment != 0;
    auto kernel = l.units > 4 ? (segmented ? conv_chain_exact_kernel<8, true> : conv_chain_exact_kernel<8, false>)
                              : (segmented ? conv_chain_exact_kernel<4, true> : conv_chain_exact_kernel<4, false>);
    int device = 0;
    cudaGetDevice(&device);
    {
        std::lock_guard<std::mutex> lock(mu);
        bool& set = done[2 * (l.units > 4) + segmented][device & 63];
        if (!set) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess) return (int)e;
            set = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(l.grid);
    cfg.blockDim = dim3(kWorkers);
    cfg.dynamicSmemBytes = (size_t)l.smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)l.p.cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return (int)cudaLaunchKernelEx(&cfg, kernel, l.p);
}

}  // namespace kn
