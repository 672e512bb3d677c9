// One to four tokens in one launch: input operation, digit planes and weight stream together.
//
// The linear of stream_planes (stream.cu) -- activations as three planes of signed 7-bit digits per 128 values with one power of two, weights
// untouched into INT8 tensor-core MMAs -- used to be two or three launches: the input operation, the digit split, the stream.  For so few
// tokens the digits of all of K fit beside the weight rings (3 bytes a value and token), so every CTA makes them for itself, each warp the
// digits of a run right before it first multiplies with them, while the weights are on their way (all digits first, then the stream: 14336 x 4096
// with SwiGLU 1.5 us slower).
//
//   weights   8 pairs of warps, each with a ring of 5 or 6 stages of 16 channels x 256 of K through TMA; each warp of a pair takes 128 of K.  The
//             shape of the boxes decides how fast the HBM streams (117 MB, nothing but the stream, us): 8 x 128 bytes 37, 16 x 128 37, 32 x
//             128 24, 128 x 128 24, 16 x 256 with sixteen rings 22.6 and with eight 21.1, 64 x 256 20.1; a plain read takes 19.7
//   digits    in shared memory, one column of the MMA for every plane of every token: columns 3 t + p for one or two tokens (one MMA where
//             stream_planes has three), 2 t, 2 t + 1 and 8 + 2 t for three or four
//   work      every CTA has an equal share of the channels, to 16; the (16 channels, 256 of K) stages of its share go round the pairs, so that
//             no K leaves warps idle
//   sums      FP32 per column, the planes of a token and then the 16 warps added in a fixed order by a 17th warp
//
// HBM-bound.  Measured on one token, kernels of a call with a cold L2, input operation + split + stream -> this: 2048 x 2048 (K x N) 5.9 -> 4.1 us,
// 5120 x 5120 15.2 -> 10, 4096 x 28672 25 -> 24.8, 14336 x 4096 with SwiGLU 18.5 -> 16.5 (a plain read of its weights: 11); MLP of one token,
// 4096 x 14336, SwiGLU, a pass among others 44.6 -> 40.3 us.  With four tokens of 4096 values and some 1000 channels the digits that every CTA makes are most
// of the time (in a graph 6.3 us, split and stream_planes 5.6; called one by one the second launch costs more than that).
#include "tc_ptx.cuh"

namespace wq {

constexpr int kFewWarps = 16, kFewPairs = 8, kFewThreads = 32 * (kFewWarps + 1), kFewRows = 16, kFewRun = 128, kFewSegment = 256, kFewSets = 3;
constexpr int kFewStageBytes = kFewRows * kFewSegment, kFewMinStages = 5, kFewMaxStages = 6, kFewBarrierBytes = 8 * (kFewPairs * kFewMaxStages + 2 * kFewSets) + 16;
constexpr int kFewMaxTokens = 4, kFewJobs = 8;
constexpr long long kFewWaitLimit = 2000000000ll;
__device__ int g_few_status = 0;

struct FewParams {
    const void* x;
    int64_t ldx;
    const float* sw;
    const void* bias;
    const void* residual;
    const void* rscale;
    void* y;
    int m, n, k, stages;
};

// Shared memory: rings, digits (runs, 3 m columns, 128 bytes), column scales (runs, 16 floats), partial sums (kFewSets sets, 16 warps, m,
// 16 rows + 1), barriers (full: 8 pairs of kFewMaxStages; sums ready, sums free: kFewSets each), the abort flag
static __host__ __device__ int few_digit_bytes(int m, int k) { return k / kFewRun * 3 * m * kFewRun; }
static __host__ __device__ int few_scale_bytes(int k) { return k / kFewRun * 16 * 4; }
static __host__ __device__ int few_partial_bytes(int m) { return kFewSets * kFewWarps * m * (kFewRows + 1) * 4; }

WQ_DEVICE bool few_wait(uint32_t bar, uint32_t parity, volatile int* gave_up) { return mbar_wait(bar, parity, gave_up, 1, &g_few_status, kFewWaitLimit); }

WQ_DEVICE void mma_s8(int* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The column of plane p of token t (BLOCKS column blocks of 8), and where it lies among the 3 m stored ones.
template <int BLOCKS> WQ_DEVICE int few_column(int t, int p) { return BLOCKS == 1 ? 3 * t + p : p < 2 ? 2 * t + p : 8 + 2 * t; }
template <int BLOCKS> WQ_DEVICE int few_stored(int column, int m) {  // columns without a plane read the first one: their sums are never used
    if (BLOCKS == 1) return column < 3 * m ? column : 0;
    if (column < 8) return column < 2 * m ? column : 0;
    return column & 1 || (column - 8) >> 1 >= m ? 0 : 2 * m + ((column - 8) >> 1);
}

template <class T, int ACT, int BLOCKS>
__global__ void __launch_bounds__(kFewThreads, 1) stream_few(const __grid_constant__ CUtensorMap map_w, const FewParams p) {
    extern __shared__ __align__(128) uint8_t few_smem[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int runs = p.k / kFewRun, segments = (runs + 1) / 2, stages = p.stages, m = p.m;
    uint8_t* digits = few_smem + kFewPairs * stages * kFewStageBytes;
    float* scales = reinterpret_cast<float*>(digits + few_digit_bytes(m, p.k));
    float* partial = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(scales) + few_scale_bytes(p.k));
    uint8_t* barriers = reinterpret_cast<uint8_t*>(partial) + few_partial_bytes(m);
    const uint32_t all_bars = smem_u32(barriers), sums_ready = all_bars + 8 * kFewPairs * kFewMaxStages, sums_free = sums_ready + 8 * kFewSets;
    volatile int* gave_up = reinterpret_cast<volatile int*>(barriers + kFewBarrierBytes - 4);
    if (threadIdx.x == 0) {
        *gave_up = 0;
        prefetch_tensormap(&map_w);
    } else if (warp == 0 || warp == 1) {  // (one thread would spend a microsecond on them)
        for (int s = int(threadIdx.x) - 1; s < kFewPairs * kFewMaxStages + 2 * kFewSets; s += 63) {
            const bool ready = s >= kFewPairs * kFewMaxStages && s < kFewPairs * kFewMaxStages + kFewSets;
            mbar_init(all_bars + 8 * s, ready ? kFewWarps : 1);
        }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    // Nothing is read before the kernel before this one has finished (it may have written the activations, and the weights as well); with that the
    // next one may be set up as this one's CTAs leave.
    dependency_wait();
    dependents_may_start();

    // this CTA's channels: items of 16, shared out evenly
    const int units = (p.n + kFewRows - 1) / kFewRows;
    const int first_item = int((long long)blockIdx.x * units / gridDim.x), items = int((long long)(blockIdx.x + 1) * units / gridDim.x) - first_item;
    const int first_row = first_item * kFewRows;
    const T* residual = static_cast<const T*>(p.residual);

    if (warp == kFewWarps) {
        // ---------------- reducer: the 16 warps' sums of an item in warp order; scales, bias, residual, one rounding ----------------
        const T* bias = static_cast<const T*>(p.bias);
        const T* rscale = static_cast<const T*>(p.rscale);
        T* y = static_cast<T*>(p.y);
        bool ok = true;
        for (int item = 0; item < items && ok; ++item) {
            const int set = item % kFewSets;
            // lane: row lane % 16 of tokens lane / 16, lane / 16 + 2; what the sums are combined with is fetched ahead of them
            const int row = lane & (kFewRows - 1), channel = first_row + item * kFewRows + row;
            const bool inside = channel < p.n;
            const float scale = inside ? p.sw[channel] : 0.f, b = inside && bias ? as_float(bias[channel]) : 0.f;
            const float rs = inside && rscale ? as_float(rscale[channel]) : 1.f;
            float before[kFewMaxTokens / 2];
#pragma unroll
            for (int i = 0; i < kFewMaxTokens / 2; ++i) {
                const int token = (lane >> 4) + 2 * i;
                before[i] = residual && inside && token < m ? as_float(residual[int64_t(token) * p.n + channel]) : 0.f;
            }
            if (!(ok = whole_warp(few_wait(sums_ready + 8 * set, uint32_t(item / kFewSets) & 1u, gave_up)))) break;
#pragma unroll
            for (int i = 0; i < kFewMaxTokens / 2; ++i) {
                const int token = (lane >> 4) + 2 * i;
                if (token < m && inside) {
                    float sum = 0.f;
#pragma unroll
                    for (int part = 0; part < kFewWarps; ++part) sum += partial[((set * kFewWarps + part) * m + token) * (kFewRows + 1) + row];
                    float v = fmaf(sum, scale, b);
                    if (residual) v = fmaf(v, rs, before[i]);
                    y[int64_t(token) * p.n + channel] = round_one<T>(v);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sums_free + 8 * set);
        }
        return;
    }

    // ---------------- streaming warps ----------------
    const int pair = warp >> 1, part = warp & 1;
    const uint8_t* ring = few_smem + pair * stages * kFewStageBytes;
    const uint32_t ring_address = smem_u32(ring), bars = all_bars + 8 * pair * kFewMaxStages;
    const bool leader = part == 0 && elect_one();  // of a pair, requests its stages
    // stages of the share are numbered item by item, segment by segment; this pair has every eighth
    int ask_item = 0, ask_segment = pair, ask_slot = 0;
    uint32_t fills = 0;  // bit s: parity of the number of fills of stage s
    auto settle = [&]() {
        while (ask_segment >= segments && ask_item < items) { ask_segment -= segments; ++ask_item; }
    };
    settle();
    auto request = [&]() {
        if (leader) {
            mbar_expect_tx(bars + 8 * ask_slot, kFewStageBytes);  // rows past N and bytes past K arrive as zeros, and count
            tma_load_2d(ring_address + ask_slot * kFewStageBytes, &map_w, bars + 8 * ask_slot, ask_segment * kFewSegment, first_row + ask_item * kFewRows);
        }
        fills ^= 1u << ask_slot;
        ask_segment += kFewPairs;
        settle();
        if (++ask_slot == stages) ask_slot = 0;
    };

    // The activations of this warp's runs of the first item, four values a lane; a job is a (run, token).  Their loads go out first: behind the rings'
    // first fill they would wait until that has drained, 3 us and more.
    uint2 raw[kFewJobs], raw_value[ACT == kActSwiglu ? kFewJobs : 1];
    {
        const T* x = static_cast<const T*>(p.x);
        int run = 2 * pair + part, token = 0;
#pragma unroll
        for (int i = 0; i < kFewJobs; ++i) {
            raw[i] = make_uint2(0u, 0u);
            if constexpr (ACT == kActSwiglu) raw_value[i] = make_uint2(0u, 0u);
            if (run < runs) {
                const T* at = x + int64_t(token) * p.ldx + run * kFewRun + 4 * lane;
                raw[i] = load_8(at);
                if constexpr (ACT == kActSwiglu) raw_value[i] = load_8(at + p.k);
                if (++token == m) { token = 0; run += kFewWarps; }
            }
        }
    }
    for (int s = 0; s < stages && ask_item < items; ++s) request();
    // the digits of one job: the input operation, rounded to T; the power of two of the run; three planes
    auto split = [&](int run, int token) {
        float v[4];
        unpack_pair<T>(raw[0].x, v[0], v[1]);
        unpack_pair<T>(raw[0].y, v[2], v[3]);
        if constexpr (ACT != kActNone) {
            float u[4] = {0.f, 0.f, 0.f, 0.f};
            if constexpr (ACT == kActSwiglu) {
                unpack_pair<T>(raw_value[0].x, u[0], u[1]);
                unpack_pair<T>(raw_value[0].y, u[2], u[3]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = as_float(round_one<T>(ACT == kActSwiglu ? silu_times(v[j], u[j]) : gelu_tanh(v[j])));
        }
#pragma unroll
        for (int i = 0; i + 1 < kFewJobs; ++i) {  // the next job's values move up: the loop over the jobs needs no copy of the code for each
            raw[i] = raw[i + 1];
            if constexpr (ACT == kActSwiglu) raw_value[i] = raw_value[i + 1];
        }
        float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
        // amax < 2^E; v / 2^(E-21) rounded to nearest is an integer of 22 bits, its upper 8 the first digit, the two groups of 7 below it the others:
        // the same value as split_planes' digits (whose first two truncate toward zero) in a third of the instructions
        const int exponent = max(int(__float_as_uint(amax) >> 23) - 126, -110);
        const float down = __uint_as_float(uint32_t(134 - exponent) << 23), up = amax > 0.f ? __uint_as_float(uint32_t(exponent + 120) << 23) : 0.f;
        uint32_t whole[4], packed[3];
#pragma unroll
        for (int j = 0; j < 4; ++j) whole[j] = uint32_t(__float2int_rn(v[j] * down * 16384.f));
        packed[0] = low_bytes(whole[0] >> 14, whole[1] >> 14, whole[2] >> 14, whole[3] >> 14);
        packed[1] = low_bytes(whole[0] >> 7, whole[1] >> 7, whole[2] >> 7, whole[3] >> 7) & 0x7f7f7f7fu;
        packed[2] = low_bytes(whole[0], whole[1], whole[2], whole[3]) & 0x7f7f7f7fu;
#pragma unroll
        for (int plane = 0; plane < 3; ++plane) {
            // the two halves of 64 swap places in every other column: the readers' 16-byte pieces of neighbouring columns use other banks
            const int column = few_column<BLOCKS>(token, plane), at = few_stored<BLOCKS>(column, m);
            *reinterpret_cast<uint32_t*>(digits + (run * 3 * m + at) * kFewRun + ((4 * lane) ^ (at & 1 ? 64 : 0))) = packed[plane];
            if (lane == 0) scales[run * 16 + column] = up * (plane == 0 ? 1.f : plane == 1 ? 1.f / 128.f : 1.f / 16384.f);
        }
    };

    int stored[BLOCKS];
#pragma unroll
    for (int block = 0; block < BLOCKS; ++block) stored[block] = few_stored<BLOCKS>(8 * block + g, m);
    bool ok = true;
    int slot = 0, segment = pair;  // this pair's first segment of the item in hand
    uint32_t parity = 0;
    for (int item = 0; item < items; ++item) {
        float acc[BLOCKS][4];
#pragma unroll
        for (int block = 0; block < BLOCKS; ++block) acc[block][0] = acc[block][1] = acc[block][2] = acc[block][3] = 0.f;
        for (; segment < segments; segment += kFewPairs) {
            const int run = 2 * segment + part;
            if (item == 0 && run < runs) {  // the run's digits, right before their first use
                for (int token = 0; token < m; ++token) split(run, token);
                __syncwarp();
            }
            if (ok) ok = whole_warp(few_wait(bars + 8 * slot, parity, gave_up));
            if (ok && run < runs) {
                const uint8_t* stage = ring + slot * kFewStageBytes + part * kFewRun;
                int sums[BLOCKS][2][4];  // (two chains of MMAs)
#pragma unroll
                for (int block = 0; block < BLOCKS; ++block)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sums[block][0][e] = sums[block][1][e] = 0;
#pragma unroll
                for (int piece = 0; piece < 2; ++piece) {
                    const uint4 row0 = *reinterpret_cast<const uint4*>(stage + g * kFewSegment + piece * 64 + 16 * t);
                    const uint4 row1 = *reinterpret_cast<const uint4*>(stage + (g + 8) * kFewSegment + piece * 64 + 16 * t);
#pragma unroll
                    for (int block = 0; block < BLOCKS; ++block) {
                        const uint4 d = *reinterpret_cast<const uint4*>(digits + (run * 3 * m + stored[block]) * kFewRun + ((piece ^ (stored[block] & 1)) * 64) + 16 * t);
                        mma_s8(sums[block][piece], row0.x, row1.x, row0.y, row1.y, d.x, d.y);
                        mma_s8(sums[block][piece], row0.z, row1.z, row0.w, row1.w, d.z, d.w);
                    }
                }
                // exact INT32 sums of the run (below 2^21 in magnitude), scaled by the token's power of two and the plane's
#pragma unroll
                for (int block = 0; block < BLOCKS; ++block) {
                    const float2 scale = *reinterpret_cast<const float2*>(scales + run * 16 + 8 * block + 2 * t);
                    acc[block][0] = fmaf(float(sums[block][0][0] + sums[block][1][0]), scale.x, acc[block][0]);
                    acc[block][1] = fmaf(float(sums[block][0][1] + sums[block][1][1]), scale.y, acc[block][1]);
                    acc[block][2] = fmaf(float(sums[block][0][2] + sums[block][1][2]), scale.x, acc[block][2]);
                    acc[block][3] = fmaf(float(sums[block][0][3] + sums[block][1][3]), scale.y, acc[block][3]);
                }
            }
            // both warps of the pair have read the stage (one that gave up comes here as well): it takes the one `stages` ahead
            asm volatile("bar.sync %0, 64;" ::"r"(2 + pair) : "memory");
            if (ok && ask_item < items) request();
            if (++slot == stages) { slot = 0; parity ^= 1u; }
        }
        segment -= segments;
        // from the second item on the pairs have other runs, unless their number divides evenly: all digits have to be there
        if (item == 0 && segments % kFewPairs) asm volatile("bar.sync 1, %0;" ::"n"(32 * kFewWarps) : "memory");
        // the planes of a token: lane t has columns 2 t and 2 t + 1 of rows g and g + 8
        float low, high;
        int token;
        if constexpr (BLOCKS == 1) {
            // token 0: columns 0, 1 (lane 0), 2 (lane 1); token 1: 3 (lane 1), 4, 5 (lane 2)
            const float pair_low = acc[0][0] + acc[0][1], pair_high = acc[0][2] + acc[0][3];
            const float next_low = __shfl_down_sync(0xffffffffu, t == 1 ? acc[0][0] : pair_low, 1), next_high = __shfl_down_sync(0xffffffffu, t == 1 ? acc[0][2] : pair_high, 1);
            low = t == 0 ? pair_low + next_low : acc[0][1] + next_low;
            high = t == 0 ? pair_high + next_high : acc[0][3] + next_high;
            token = t;
        } else {
            low = acc[0][0] + acc[0][1] + acc[1][0];
            high = acc[0][2] + acc[0][3] + acc[1][2];
            token = t;
        }
        const int set = item % kFewSets;
        if (ok && item >= kFewSets) ok = whole_warp(few_wait(sums_free + 8 * set, uint32_t(item / kFewSets - 1) & 1u, gave_up));
        if (ok) {
            if (token < m) {
                float* mine = partial + ((set * kFewWarps + warp) * m + token) * (kFewRows + 1);
                mine[g] = low;
                mine[g + 8] = high;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sums_ready + 8 * set);
        }
    }
    if (!ok && part == 0) await_issued_fills(bars, stages, fills);
}

// ---- host side -------------------------------------------------------------------------------------------------------
static int few_bytes(int m, int k, int stages) {
    return kFewPairs * stages * kFewStageBytes + few_digit_bytes(m, k) + few_scale_bytes(k) + few_partial_bytes(m) + kFewBarrierBytes;
}

// The digits of all of K beside the weight rings, and the activations of a warp's runs in its registers: up to 16384 values for one token, 8192
// for two, 4096 for three and four.
bool stream_few_takes(int m, int k) {
    return m >= 1 && m <= kFewMaxTokens && k > 0 && k % kFewRun == 0 && (k / kFewRun + kFewWarps - 1) / kFewWarps * m <= kFewJobs &&
           few_bytes(m, k, kFewMinStages) <= 227 * 1024;
}

template <class T, int ACT, int BLOCKS>
static int launch_few_shape(const int8_t* w, const FewParams& p, int sms, cudaStream_t stream) {
    auto kernel = stream_few<T, ACT, BLOCKS>;
    static bool configured[64] = {};  // the attribute belongs to a device's copy of the kernel
    int device = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64 || !configured[device]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return int(e);
        if (device >= 0 && device < 64) configured[device] = true;
    }
    CUtensorMap map_w;
    if (!make_byte_matrix_map(&map_w, w, p.n, p.k, kFewSegment, kFewRows)) return int(cudaErrorNotSupported);
    const int units = (p.n + kFewRows - 1) / kFewRows, ctas = units < sms ? units : sms;
    const cudaError_t launched = launch_after_previous(kernel, dim3(ctas), dim3(kFewThreads), size_t(few_bytes(p.m, p.k, p.stages)), stream, map_w, p);
    return int(launched != cudaSuccess ? launched : cudaGetLastError());
}

template <class T, int ACT> static int launch_few_act(const int8_t* w, const FewParams& p, int sms, cudaStream_t stream) {
    return p.m <= 2 ? launch_few_shape<T, ACT, 1>(w, p, sms, stream) : launch_few_shape<T, ACT, 2>(w, p, sms, stream);
}

template <class T> static int launch_few(const int8_t* w, const FewParams& p, int act, int sms, cudaStream_t stream) {
    if (act == kActNone) return launch_few_act<T, kActNone>(w, p, sms, stream);
    if (act == kActSwiglu) return launch_few_act<T, kActSwiglu>(w, p, sms, stream);
    if (act == kActGelu) return launch_few_act<T, kActGelu>(w, p, sms, stream);
    return -2;
}

// x: (m, K) rows, SwiGLU (m, 2 K); 8-byte aligned, ldx a multiple of 4; w 16-byte aligned; a shape that stream_few_takes().
int stream_few_launch(const void* x, int64_t ldx, const int8_t* w, const float* sw, const void* bias, const void* residual, const void* rscale, void* y, int m,
                      int n, int k, int dtype, int act, int sms, cudaStream_t stream) {
    if (!stream_few_takes(m, k)) return -2;
    const int stages = few_bytes(m, k, kFewMaxStages) <= 227 * 1024 ? kFewMaxStages : kFewMinStages;
    const FewParams p{x, ldx, sw, bias, residual, rscale, y, m, n, k, stages};
    if (sms <= 0) sms = 148;
    if (dtype == 0) return launch_few<__half>(w, p, act, sms, stream);
    if (dtype == 1) return launch_few<bf16>(w, p, act, sms, stream);
    return -1;
}

int stream_few_status_take() {
    int code = 0;
    const int zero = 0;
    if (cudaMemcpyFromSymbol(&code, g_few_status, sizeof(int)) != cudaSuccess) return -1;
    if (code) cudaMemcpyToSymbol(g_few_status, &zero, sizeof(int));
    return code;
}

}  // namespace wq
