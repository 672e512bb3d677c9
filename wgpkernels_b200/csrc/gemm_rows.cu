// INT8 GEMM of `row` and `exact` for up to 128 rows on tcgen05: clusters of CTAs share the K of a tile of 128 output channels.
//
// With so few rows the tiles of gemm_i8_tc leave most SMs idle (64 x 5120 x 5120: 80 CTAs of 64 channels, each bringing in all of A), and the call
// takes what one CTA needs for all of K.  Here the weights are the M x K operand (128 channels fill the tensor-memory lanes whatever the rows),
// the activations the N x K one (hi rows, then lo rows: one MMA for both parts), and a cluster of 2 to 8 CTAs splits K:
//
//   warp 0      TMA producer: {128 x 128 bytes of W, rows x 128 of A, [rows x 128 of A_lo]} per block of K, 128-byte swizzle, no multicast
//   warp 1      MMA issue (one elected lane): all blocks of the CTA's share into one accumulator in tensor memory
//   warp 2      owns tensor memory
//   warps 4-7   the INT32 sums from tensor memory to the CTA of the cluster that finishes their rows, through distributed shared memory
//   all warps   the CTA's share of the rows: integer sums over the cluster (exact, so the order does not matter), scales, bias, residual, store
//
// The outputs are the bits of gemm_i8_tc.  Bound by latency: launch, first bytes, two cluster barriers and the exchange take 5.5 us with a few rows
// and 9 with 128, the stream of the weights the rest.  Measured (`exact`, L2 cold, gemm_i8_tc -> this, us): 64 x 5120 x 5120 (rows x channels
// x K) 18.6 -> 11.9, 29 x 5120 x 5120 18.4 -> 10.9, 64 x 1024 x 14336 42.0 -> 10.9, 48 x 2048 x 2048 10.0 -> 7.4, 128 x 5120 x 5120
// 18.4 -> 16.3.  (Four-byte stores to the other CTAs instead of sixteen: 13.8 on the first of these, 19.3 on the last.)
//
// Every wait is bounded; a wait that gives up raises the CTA's abort flag, and every thread still comes to the cluster's two barriers.
#include <cuda.h>

#include "tc_ptx.cuh"

namespace wq {

constexpr int kRowsThreads = 256, kRowsMost = 128, kRowsChannels = 128, kRowsMaxStages = 8, kRowsBarrierBytes = 192 + 4 * kRowsMost;
constexpr int kRowsRoom = 226 * 1024 - kRowsBarrierBytes;
constexpr long long kRowsWaitLimit = 4000000000ll;
__device__ int g_rows_status = 0;

struct RowsParams {
    const float* sa;
    const float* sw;
    const void* bias;
    const void* residual;
    const void* rscale;
    void* y;
    int64_t ld_y, ld_residual;
    int m, n, kblocks, slots, stages, columns;  // slots: m rounded up to 16; columns: of tensor memory
};

// one lane's answer: to be put through whole_warp() before the warp acts on it
WQ_DEVICE bool rows_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    return mbar_wait(bar, parity, abort_flag, code, &g_rows_status, kRowsWaitLimit);
}

template <class T, bool HILO>
__global__ void __launch_bounds__(kRowsThreads, 1)
gemm_few_rows(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_lo, const RowsParams p) {
    constexpr int kParts = HILO ? 2 : 1, kWeightBytes = kRowsChannels * kStageK;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int part_bytes = p.slots * kStageK, stage_bytes = kWeightBytes + kParts * part_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kRowsRoom);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kRowsMaxStages, bar_sums = bar_empty + 8 * kRowsMaxStages;
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(bars) + 160);
    int& abort_word = *reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 164);
    volatile int* abort_flag = &abort_word;
    float* row_scales = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 192);
    if (threadIdx.x == 0) {
        abort_word = 0;
        if (smem_u32(smem) & 1023u) {  // the swizzle of the operand stages needs it: reported, nothing computed
            abort_word = kStatusSharedAlignment;
            atomicCAS(&g_rows_status, 0, int(kStatusSharedAlignment));
        }
        for (int s = 0; s < kRowsMaxStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_sums, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_a);
        if (HILO) prefetch_tensormap(&map_lo);
    }
    if (warp == 2) tmem_alloc(smem_u32(&tmem_slot), p.columns);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    // launched behind the kernel before it on the stream: everything from here on may have been written by it
    dependency_wait();

    const int ranks = int(cluster_size()), rank = int(cluster_rank()), tile = blockIdx.x / ranks;
    const int kb0 = rank * p.kblocks / ranks, blocks = (rank + 1) * p.kblocks / ranks - kb0;
    bool ok = *abort_flag == 0;

    if (warp == 0 && ok) {
        // ---------------- TMA producer ----------------
        const bool leader = elect_one();
        int stage = 0;
        uint32_t fills = 0;  // bit s: parity of the number of fills of stage s
        for (int b = 0; b < blocks; ++b) {
            if (!(ok = whole_warp(rows_wait(bar_empty + 8 * stage, ((fills >> stage) & 1u) ^ 1u, abort_flag, kTimeoutEmpty)))) break;
            fills ^= 1u << stage;
            if (leader) {
                const uint32_t dst = smem_u32(smem + stage * stage_bytes), full = bar_full + 8 * stage;
                const int x = (kb0 + b) * kStageK;
                mbar_expect_tx(full, stage_bytes);  // what lies past N, M or K arrives as zeros, and counts
                tma_load_2d(dst, &map_w, full, x, tile * kRowsChannels);
                tma_load_2d(dst + kWeightBytes, &map_a, full, x, 0);
                if (HILO) tma_load_2d(dst + kWeightBytes + part_bytes, &map_lo, full, x, 0);
            }
            if (++stage == p.stages) stage = 0;
        }
        // Whatever became of the waits, this one's or the issuer's: no copy is in flight when the stages become the place of the sums, or when the CTA
        // leaves.  (The issuer waits for the same copies.)
        await_issued_fills(bar_full, p.stages, fills);
    } else if (warp == 1 && ok) {
        // ---------------- MMA issuer ----------------
        const bool leader = elect_one();
        const uint32_t idesc = instruction_descriptor(p.slots * kParts);
        int stage = 0;
        uint32_t phase = 0;
        for (int b = 0; b < blocks; ++b) {
            if (!whole_warp(rows_wait(bar_full + 8 * stage, phase, abort_flag, kTimeoutFull))) break;
            tc_fence_after();
            if (leader) {
                const uint32_t address = smem_u32(smem + stage * stage_bytes);
                const uint64_t w_desc = smem_descriptor(address), a_desc = smem_descriptor(address + kWeightBytes);
#pragma unroll
                for (int j = 0; j < kStageK / kMmaK; ++j) {
                    const uint64_t step = uint64_t(j * kMmaK >> 4);
                    mma_i8(tmem_base, w_desc + step, a_desc + step, idesc, b == 0 && j == 0 ? 0u : 1u);
                }
                tc_commit(bar_empty + 8 * stage);
                if (b == blocks - 1) tc_commit(bar_sums);
            }
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
    } else if (warp == 3) {
        for (int row = lane; row < p.m; row += 32) row_scales[row] = p.sa[row];
    } else if (warp >= 4 && ok) {
        whole_warp(rows_wait(bar_sums, 0u, abort_flag, kTimeoutTmemFull));
    }
    // Every MMA of the cluster has read its operands (or its CTA has given up): the stages become the place where the sums are exchanged.
    __syncwarp();
    cluster_sync();

    // Rows go to the CTAs of the cluster in runs of `share`, a multiple of four; a CTA finds the sums of its rows as (source CTA, four rows, part,
    // channel, row of the four), so that a lane sends and fetches sixteen bytes.
    const int quads = (p.slots / 4 + ranks - 1) / ranks, share = 4 * quads;
    constexpr int kQuadBytes = kRowsChannels * 16;
    const bool complete = *abort_flag == 0;  // (of this CTA; a wait that gave up leaves unspecified outputs and a status)
    if (warp >= 4 && complete) {  // (all eight warps: up to 4 % faster with 128 rows, 5 % slower with 33)
        tc_fence_after();
        const int quarter = warp & 3;
        const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16);
        const uint32_t mine = smem_u32(smem) + rank * quads * kParts * kQuadBytes + (quarter * 32 + lane) * 16;
        for (int c0 = 0; c0 < p.slots * kParts; c0 += 16) {
            int sums[16];
            tmem_load_16(taddr + c0, sums);
            tmem_load_wait();
            tmem_loaded(sums);
            const int part = c0 >= p.slots ? 1 : 0, quad0 = (c0 - part * p.slots) / 4;
            int owner = quad0 / quads, within = quad0 - owner * quads;
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(in_cta(mine, uint32_t(owner)) + (within * kParts + part) * kQuadBytes), "r"(sums[j]),
                             "r"(sums[j + 1]), "r"(sums[j + 2]), "r"(sums[j + 3])
                             : "memory");
                if (++within == quads) {
                    within = 0;
                    ++owner;
                }
            }
        }
        tc_fence_before();
    }
    // the channel's parameters are on their way while the cluster meets
    const int channel = threadIdx.x & (kRowsChannels - 1), column = tile * kRowsChannels + channel;
    const bool inside = column < p.n;
    const T* bias = static_cast<const T*>(p.bias);
    const T* residual = inside ? static_cast<const T*>(p.residual) : nullptr;
    const T* rscale = static_cast<const T*>(p.rscale);
    const float scale = inside ? p.sw[column] : 0.f, offset = inside && bias ? as_float(bias[column]) : 0.f, rs = inside && rscale ? as_float(rscale[column]) : 1.f;
    __syncwarp();
    cluster_sync();

    // ---------------- the CTA's rows: two threads a channel, four rows at a time ----------------
    if (complete && inside) {
        T* y = static_cast<T*>(p.y);
        constexpr int kStep = kRowsThreads / kRowsChannels;
        const int first = rank * share, end = min(first + share, p.m);
        auto fetch = [&](int quad, float* before) {  // (the residual of four rows, a step ahead)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = first + 4 * quad + e;
                before[e] = residual && row < end ? as_float(residual[row * p.ld_residual + column]) : 0.f;
            }
        };
        int quad = int(threadIdx.x) / kRowsChannels;
        float before[4], next[4];
        fetch(quad, before);
        for (; first + 4 * quad < end; quad += kStep) {
            fetch(quad + kStep, next);
            int high[4] = {0, 0, 0, 0}, low[4] = {0, 0, 0, 0};
            const uint8_t* at = smem + quad * kParts * kQuadBytes + channel * 16;
            for (int source = 0; source < ranks; ++source, at += quads * kParts * kQuadBytes) {
                const int4 h = *reinterpret_cast<const int4*>(at);
                high[0] += h.x; high[1] += h.y; high[2] += h.z; high[3] += h.w;
                if (HILO) {
                    const int4 l = *reinterpret_cast<const int4*>(at + kQuadBytes);
                    low[0] += l.x; low[1] += l.y; low[2] += l.z; low[3] += l.w;
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = first + 4 * quad + e;
                if (row < end) {
                    float v = float(high[e]);
                    if (HILO) v = fmaf(float(low[e]), 1.f / 254.f, v);
                    v = fmaf(v * row_scales[row], scale, offset);
                    if (residual) v = fmaf(v, rs, before[e]);
                    y[row * p.ld_y + column] = round_one<T>(v);
                }
                before[e] = next[e];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.columns);
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------
bool make_swizzled_byte_map(CUtensorMap* map, const void* base, int64_t rows, int k, int box_rows);  // gemm_tc.cu

// Clusters of `ctas` CTAs of this kernel (one an SM) that the current GPU holds at once: its SMs come in groups that no cluster crosses.
static int clusters_at_once(int ctas) {
    static int known[64][9] = {};  // 0: not asked yet (the answer plus one is kept; threads that ask at the same time write the same)
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64 || ctas < 1 || ctas > 8) return 0;
    if (!known[device][ctas]) {
        auto kernel = gemm_few_rows<bf16, true>;
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(unsigned(ctas));
        config.blockDim = dim3(kRowsThreads);
        config.dynamicSmemBytes = kRowsRoom + kRowsBarrierBytes;
        cudaLaunchAttribute attribute;
        attribute.id = cudaLaunchAttributeClusterDimension;
        attribute.val.clusterDim.x = unsigned(ctas);
        attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
        config.attrs = &attribute;
        config.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsRoom + kRowsBarrierBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
            (void)cudaGetLastError();
            clusters = 0;
        }
        known[device][ctas] = clusters + 1;
    }
    return known[device][ctas] - 1;
}

// CTAs of a cluster for this product, 0 when it is not this kernel's: as many as the SMs hold for all tiles at once.
int gemm_few_rows_cluster(int m, int n, int k, int sms) {
    if (m < 1 || m > kRowsMost || n < 1 || k < 1) return 0;
    if (sms <= 0) sms = 148;
    const int tiles = (n + kRowsChannels - 1) / kRowsChannels, kblocks = (k + kStageK - 1) / kStageK;
    for (int ctas = 8; ctas >= 2; --ctas)
        if (ctas <= kblocks && tiles * ctas <= sms && tiles <= clusters_at_once(ctas)) return ctas;
    return 0;
}

// Whether this kernel is the faster one (against gemm_i8_tc, which has tiles of 64 channels for the shapes that fit clusters).  gemm_i8_tc brings all
// of K into one SM; here a CTA has its share of K, the exchange costs by the rows (the more where a CTA has two blocks of K or fewer to hide
// its start behind), and all rows go to every CTA; both stream the weights.  In ns, fitted to 9 x 13 x 8 sizes (17 to 128 rows, 512 to 15360 channels, K
// of 1024 to 14336) and taken where it wins by a twentieth.  Near the line (gemm_i8_tc and this, us): `row` 96 x 9216 x 4096 (rows x channels x K)
// 13.1 and 14.1, 128 x 5120 x 4096 12.3 and 12.7, 96 x 512 x 1536 6.1 and 6.7 (left alone), 48 x 9216 x 2048 10.8 and 9.1; `exact` 33 x 3072 x
// 1024 7.6 and 7.0.
bool gemm_few_rows_wins(int m, int n, int k, bool hilo, int sms) {
    const int64_t ctas = gemm_few_rows_cluster(m, n, k, sms), slots = (m + 15) / 16 * 16, tiles = (n + kRowsChannels - 1) / kRowsChannels;
    if (!ctas) return false;
    const double kilo = k / 1000., share = kilo / ctas, weights = kilo * n / 1000., copies = double(slots * tiles * ctas) / (sms > 0 ? sms : 148);
    const double start = k <= 2 * kStageK * ctas ? 5. * slots : 0.;
    const double whole = hilo ? 4530 + (2490 - 1.4 * m) * kilo + 79.2 * weights : 4370 + (1651 - 1.5 * m) * kilo + 73.5 * weights;
    const double split = hilo ? 4050 + 29.9 * slots + (1220 + 4.64 * slots) * share + 84.7 * weights + 23.1 * copies
                              : 3970 + 15.4 * slots + (1234 + 0.75 * slots) * share + 97.9 * weights + 25.5 * copies;
    return split + start < 0.95 * whole;
}

template <class T, bool HILO>
static int launch_rows_kernel(const int8_t* a, const int8_t* a_lo, const int8_t* w, RowsParams& p, int k, int ctas, cudaStream_t stream) {
    auto kernel = gemm_few_rows<T, HILO>;
    constexpr int kParts = HILO ? 2 : 1;
    static bool configured[64] = {};  // the attribute belongs to a device's copy of the kernel
    int device = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64 || !configured[device]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsRoom + kRowsBarrierBytes);
        if (e != cudaSuccess) return int(e);
        if (device >= 0 && device < 64) configured[device] = true;
    }
    p.slots = (p.m + 15) / 16 * 16;
    const int stages = kRowsRoom / (kRowsChannels * kStageK + kParts * p.slots * kStageK);
    p.stages = stages > kRowsMaxStages ? kRowsMaxStages : stages;
    p.columns = 32;
    while (p.columns < p.slots * kParts) p.columns *= 2;
    p.kblocks = (k + kStageK - 1) / kStageK;
    CUtensorMap map_w, map_a, map_lo;
    if (!make_swizzled_byte_map(&map_w, w, p.n, k, kRowsChannels) || !make_swizzled_byte_map(&map_a, a, p.m, k, p.slots)) return int(cudaErrorNotSupported);
    map_lo = map_a;
    if (HILO && !make_swizzled_byte_map(&map_lo, a_lo, p.m, k, p.slots)) return int(cudaErrorNotSupported);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(unsigned((p.n + kRowsChannels - 1) / kRowsChannels * ctas));
    config.blockDim = dim3(kRowsThreads);
    config.dynamicSmemBytes = kRowsRoom + kRowsBarrierBytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = unsigned(ctas);
    attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
    config.attrs = attributes;
    config.numAttrs = 2;
    const cudaError_t launched = cudaLaunchKernelEx(&config, kernel, map_w, map_a, map_lo, p);
    return int(launched != cudaSuccess ? launched : cudaGetLastError());
}

// a_lo: `exact`, else `row`.  a, a_lo and w 16-byte aligned.
int gemm_few_rows_launch(const int8_t* a, const int8_t* a_lo, const float* sa, const int8_t* w, const float* sw, const void* bias, const void* residual,
                         const void* rscale, void* y, int64_t ld_y, int64_t ld_residual, int m, int n, int k, bool is_bf16, int sms, cudaStream_t stream) {
    const int ctas = gemm_few_rows_cluster(m, n, k, sms);
    if (!ctas || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(a_lo) | reinterpret_cast<uintptr_t>(w)) & 15)) return -2;
    RowsParams p{sa, sw, bias, residual, rscale, y, ld_y, ld_residual, m, n, 0, 0, 0, 0};
    if (is_bf16) return a_lo ? launch_rows_kernel<bf16, true>(a, a_lo, w, p, k, ctas, stream) : launch_rows_kernel<bf16, false>(a, a_lo, w, p, k, ctas, stream);
    return a_lo ? launch_rows_kernel<__half, true>(a, a_lo, w, p, k, ctas, stream) : launch_rows_kernel<__half, false>(a, a_lo, w, p, k, ctas, stream);
}

int gemm_rows_status_take() {
    int code = 0;
    const int zero = 0;
    if (cudaMemcpyFromSymbol(&code, g_rows_status, sizeof(int)) != cudaSuccess) return -1;
    if (code) cudaMemcpyToSymbol(g_rows_status, &zero, sizeof(int));
    return code;
}

}  // namespace wq
