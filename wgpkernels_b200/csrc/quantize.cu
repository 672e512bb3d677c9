// Activation preparation kernels: per-(row, 128-block) INT8 quantizer, row / hi-lo INT8 quantizer, few-token transform,
// ConvRot group rotation.  All of them stream the activation once from HBM with 16-byte loads and fuse the input operation
// (rms_norm / swiglu / gelu-tanh) in FP32.  Results are bit-for-bit those of the reference library
// (wgpkernels/int8/int8_gemm.cu:253-485, 1814-1831 of WGPKernels): same FP32 expressions, same fixed-order reductions.
#include "common.cuh"

namespace wq {

// Row window of the *_at entry points: the input rows start at row first + counter[0] * step of x, the counter being read on the GPU
// when the kernel runs (a CUDA graph replays the launch while its loop counter advances).  No counter: row 0.
struct RowShift { const long long* counter; long long first, step; };
template <class T> WQ_DEVICE const T* first_row(const T* x, int64_t ldx, const RowShift& shift) {
    return shift.counter ? x + (shift.first + __ldg(shift.counter) * shift.step) * ldx : x;
}

// ---- one 256-element chunk -> two 128-element blocks (16 lanes each): absmax, scale, INT8 codes --------------------------
template <int GROUP, bool PAIRS = false>
WQ_DEVICE void store_chunk_as_blocks(const float* v, int lane, int64_t row, int base, int k, int kblocks, int8_t* __restrict__ q,
                                     float* __restrict__ scale) {
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));  // stays inside each half warp
    // every lane holds its block's absmax: all of them do the division (the instructions issue once per warp either way; a branch for the
    // first lane of a block and a shuffle back would only add to them), the block's first lane stores the scale
    const float inv = amax > 0.f ? 127.f / amax : 0.f;
    const int block = base / kBlockK + (lane >> 4);
    if ((lane & 15) == 0 && block < kblocks) scale[row * kblocks + block] = amax * group_norm<GROUP>() / 127.f;
    const int col = base + lane * 8;
    if (col < k) {
        int c[8];
        if constexpr (PAIRS) {  // two-wide multiplies (each half rounds as the scalar multiply does): fewer instructions where the input
                                // operation leaves registers to pair; the row kernels, short of registers, keep the scalar form
            const float2 inverse = make_float2(inv, inv);
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float2 scaled = __fmul2_rn(make_float2(v[j], v[j + 1]), inverse);
                c[j] = __float2int_rn(scaled.x);
                c[j + 1] = __float2int_rn(scaled.y);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) c[j] = __float2int_rn(v[j] * inv);
        }
        *reinterpret_cast<uint2*>(q + row * k + col) = make_uint2(pack_bytes(c[0], c[1], c[2], c[3]), pack_bytes(c[4], c[5], c[6], c[7]));
    }
}

// RMSNorm needs the row's sum of squares first: one CTA per row.  CPW > 0: the row (K <= 2048 * CPW) stays in registers, one read.
// CPW == 0: any K, the row is read twice (the second read comes from L2).
// Sum of squares: thread (warp w, lane l) accumulates fmaf(v, v, ss) over chunks w, w + 8, ... in order; then the ordered CTA sum.
template <class T, int GROUP, int CPW>
__global__ void __launch_bounds__(kRowThreads, CPW > 0 && CPW <= 4 ? 6 : 1) quantize_blocks_rms(const T* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale, int m, int k,
                                                                   int64_t ldx, const T* __restrict__ act_weight, float eps, RowShift shift) {
    __shared__ float slots[9];
    dependents_may_start();  // the GEMM behind this kernel may be set up under its tail (it waits for this grid before it reads anything)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x;
    const T* src = first_row(x, ldx, shift) + row * ldx;
    const int kblocks = (k + kBlockK - 1) / kBlockK;
    float ss = 0.f;
    if constexpr (CPW > 0) {
        static_assert(sizeof(T) == 2, "rms_norm takes 16-bit inputs");
        float v[CPW][8];
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int col = (warp + 8 * i) * kChunk + lane * 8;
            load_eight(src + col, v[i], col < k);
        }
#pragma unroll
        for (int i = 0; i < CPW; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
        const float inv_rms = cta_inverse_rms(ss, slots, k, eps);
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int base = (warp + 8 * i) * kChunk;
            if (base < k) {  // warp-uniform
                // the RMSNorm weights of the chunk come from L1 / L2 when they are needed: held from before the reduction they would cost the
                // registers that let six CTAs share an SM (the kernel is bound by instruction issue: occupancy is what it needs)
                const uint4 raw = (act_weight && base + lane * 8 < k) ? __ldg(reinterpret_cast<const uint4*>(act_weight + base + lane * 8)) : make_uint4(0u, 0u, 0u, 0u);
                float w[8];
                unpack_pair<T>(raw.x, w[0], w[1]);
                unpack_pair<T>(raw.y, w[2], w[3]);
                unpack_pair<T>(raw.z, w[4], w[5]);
                unpack_pair<T>(raw.w, w[6], w[7]);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[i][j] = v[i][j] * inv_rms * (act_weight ? w[j] : 1.f);
                rotate_chunk<GROUP>(v[i]);
                store_chunk_as_blocks<GROUP>(v[i], lane, row, base, k, kblocks, q, scale);
            }
        }
    } else {
        for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
            float v[8];
            load_eight(src + base + lane * 8, v, base + lane * 8 < k);
#pragma unroll
            for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
        }
        const float inv_rms = cta_inverse_rms(ss, slots, k, eps);
        for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
            float v[8];
            const bool valid = base + lane * 8 < k;
            load_eight(src + base + lane * 8, v, valid);
            scale_by_rms(v, inv_rms, act_weight, base + lane * 8, valid);
            rotate_chunk<GROUP>(v);
            store_chunk_as_blocks<GROUP>(v, lane, row, base, k, kblocks, q, scale);
        }
    }
}

// No row statistic: every (row, 256-element chunk) is independent.  One warp per item and nothing else: the row is the grid's y
// coordinate and the chunk comes from x, so there is no loop, no division and no bookkeeping -- the input operations (the accurate
// tanhf / expf of gelu and swiglu) are what these launches spend their time on, and every register and instruction beside them
// costs occupancy.  The host launches batches of at most 65535 rows (the grid's y limit).
template <class T, int GROUP, int ACT>
__global__ void __launch_bounds__(256) quantize_blocks_items(const T* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale, int64_t row0, int k,
                                                             int64_t ldx, RowShift shift) {
    dependents_may_start();
    const int lane = threadIdx.x & 31;
    const int base = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kChunk;
    if (base >= k) return;
    const int kblocks = (k + kBlockK - 1) / kBlockK;
    const int64_t row = row0 + blockIdx.y;
    float v[8];
    load_op<T, ACT>(first_row(x, ldx, shift) + row * ldx, k, base + lane * 8, v, base + lane * 8 < k);
    rotate_chunk<GROUP>(v);
    store_chunk_as_blocks<GROUP, true>(v, lane, row, base, k, kblocks, q, scale);
}

// ---- gelu without the accurate tanhf ----------------------------------------------------------------------------------------
// The codes and scales are those of gelu_tanh(), bit for bit, but few elements are put through it.  An approximation of gelu (two special-function
// instructions an element) gives t = v * inv to within a known bound; where no rounding boundary lies that close to t, the accurate value
// rounds to the same code.  The elements nearer to a boundary (some 1e-4 of them), and those that are not finite, are computed
// accurately.  The scale needs the block's accurate absmax: above 0.35 gelu is larger than anywhere below zero (0.17 at most) and grows with x
// by far more than its own rounding from one 16-bit value to the next, so it is the gelu of the block's largest x; one lane in four
// evaluates that, divides and stores the scale for its block.  Warps with a block that has no such x take the general path.
//   error of t: the sigmoid form x / (1 + 2^a) is within 4.5e-7 |x| of gelu (ex2 2^-22, rcp 2^-23, and |a| 1.7e-7 through the roundings of a,
//   which counts most where 2^a is about 5), gelu_tanh() within 3e-7 |x| (tanhf two units, 1 + tanhf one): 1e-6 |x| inv together, and three
//   roundings of t itself, 2.3e-5 for |t| <= 127.  (Below -6, where 1 + tanhf() is 0 or next to it, both are within 1e-9.)
// One warp takes four chunks of a row: their loads are in flight together, and what is done once per block or per warp (317 instructions a
// chunk with tanhf, 255 with this arithmetic and a chunk a warp) spreads over more elements.
// Measured (32760 x 13824, BF16): 567 us with tanhf, 350 so (2.40 and 3.88 TB/s; 1560 x 13824: 31.0 and 21.5).
constexpr float kRoundMagic = 12582912.f;  // 1.5 * 2^23: adding it rounds |t| < 2^22 to the nearest even integer, whose low byte is the sum's low byte
constexpr int kGeluChunks = 4;

WQ_DEVICE float exp2_fast(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
WQ_DEVICE float reciprocal_fast(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// The larger magnitude (with either sign), or NaN where either is.
WQ_DEVICE float magnitude_or_nan(float a, float b) {
    float r;
    asm("max.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <class T>
__global__ void __launch_bounds__(256, 5) quantize_blocks_gelu(const T* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale, int64_t row0, uint32_t items,
                                                               int k, int64_t ldx, RowShift shift) {
    dependents_may_start();
    const int lane = threadIdx.x & 31;
    const uint32_t item = blockIdx.x * 8 + (threadIdx.x >> 5), groups = uint32_t(k + kGeluChunks * kChunk - 1) / (kGeluChunks * kChunk);
    if (item >= items) return;
    const int first = int(item % groups) * (kGeluChunks * kChunk);
    const int kblocks = (k + kBlockK - 1) / kBlockK;
    const int64_t row = row0 + item / groups;
    const T* src = first_row(x, ldx, shift) + row * ldx + first + lane * 8;
    uint4 raw[kGeluChunks];
#pragma unroll
    for (int c = 0; c < kGeluChunks; ++c)
        raw[c] = first + c * kChunk + lane * 8 < k ? __ldg(reinterpret_cast<const uint4*>(src + c * kChunk)) : make_uint4(0u, 0u, 0u, 0u);
    // Largest x of every block (16 lanes of a chunk): the lanes share the chunks out as they go, so that lane l ends with chunk (l >> 2) & 3 of its half
    float largest[kGeluChunks], bound[kGeluChunks];  // bound: the |x| that counts in the error of this lane's elements
#pragma unroll
    for (int c = 0; c < kGeluChunks; ++c) {
        float smallest;
        extremes<T>(raw[c], largest[c], smallest);
        bound[c] = fmaxf(largest[c], fminf(-smallest, 6.f));
    }
    static_assert(kGeluChunks == 4, "two steps share out four chunks");
    float block_largest;
    {
        const bool upper = lane & 8, odd = lane & 4;
        const float keep0 = upper ? largest[2] : largest[0], keep1 = upper ? largest[3] : largest[1];
        const float give0 = upper ? largest[0] : largest[2], give1 = upper ? largest[1] : largest[3];
        const float pair0 = fmaxf(keep0, __shfl_xor_sync(0xffffffffu, give0, 8)), pair1 = fmaxf(keep1, __shfl_xor_sync(0xffffffffu, give1, 8));
        block_largest = fmaxf(odd ? pair1 : pair0, __shfl_xor_sync(0xffffffffu, odd ? pair0 : pair1, 4));
        block_largest = fmaxf(block_largest, __shfl_xor_sync(0xffffffffu, block_largest, 2));
        block_largest = fmaxf(block_largest, __shfl_xor_sync(0xffffffffu, block_largest, 1));
    }
    const int block = first / kBlockK + 2 * ((lane >> 2) & 3) + (lane >> 4);
    if (__any_sync(0xffffffffu, !(block_largest >= 0.35f) && block < kblocks)) {
#pragma unroll 1
        for (int c = 0; c < kGeluChunks && first + c * kChunk < k; ++c) {
            float v[8];
            load_op<T, kActGelu>(src - lane * 8, k, c * kChunk + lane * 8, v, first + c * kChunk + lane * 8 < k);
            store_chunk_as_blocks<0, true>(v, lane, row, first + c * kChunk, k, kblocks, q, scale);
        }
        return;
    }
    const float amax = gelu_tanh(block_largest), block_inv = block < kblocks ? 127.f / amax : 0.f;  // (0: what lies past K takes no accurate path)
    if ((lane & 3) == 0 && block < kblocks) scale[row * kblocks + block] = amax / 127.f;
    int8_t* dst = q + row * k + first + lane * 8;
#pragma unroll
    for (int c = 0; c < kGeluChunks; ++c) {
        if (first + c * kChunk >= k) break;
        const float inv = __shfl_sync(0xffffffffu, block_inv, (lane & 16) | (c << 2));
        const float2 inverse = make_float2(inv, inv);
        float2 x2[4], t[4], sum[4];
        unpack_pair<T>(raw[c].x, x2[0].x, x2[0].y);
        unpack_pair<T>(raw[c].y, x2[1].x, x2[1].y);
        unpack_pair<T>(raw[c].z, x2[2].x, x2[2].y);
        unpack_pair<T>(raw[c].w, x2[3].x, x2[3].y);
        float farthest = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // 2^a = exp(-2 inner): a = x (c1 + c3 x^2), c1 = -2 log2(e) sqrt(2 / pi), c3 = 0.044715 c1
            const float2 a = __fmul2_rn(x2[j], __ffma2_rn(__fmul2_rn(x2[j], x2[j]), make_float2(-0.10294324f, -0.10294324f), make_float2(-2.3022082f, -2.3022082f)));
            const float2 e = __fadd2_rn(make_float2(exp2_fast(a.x), exp2_fast(a.y)), make_float2(1.f, 1.f));
            t[j] = __fmul2_rn(__fmul2_rn(x2[j], inverse), make_float2(reciprocal_fast(e.x), reciprocal_fast(e.y)));
            sum[j] = __fadd2_rn(t[j], make_float2(kRoundMagic, kRoundMagic));
            const float2 distance = __ffma2_rn(t[j], make_float2(-1.f, -1.f), __fadd2_rn(sum[j], make_float2(-kRoundMagic, -kRoundMagic)));
            farthest = magnitude_or_nan(farthest, magnitude_or_nan(distance.x, distance.y));
        }
        const uint32_t* bits = reinterpret_cast<const uint32_t*>(sum);
        uint2 codes = make_uint2(low_bytes(bits[0], bits[1], bits[2], bits[3]), low_bytes(bits[4], bits[5], bits[6], bits[7]));
        const float far_enough = 0.5f - 3e-5f - 1e-6f * inv * bound[c];
        if (!(fabsf(farthest) < far_enough)) {  // (or not a number)
            uint32_t word[2] = {codes.x, codes.y};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float tj = j & 1 ? t[j / 2].y : t[j / 2].x;
                if (!(fabsf(tj - rintf(tj)) < far_enough)) {
                    const int code = __float2int_rn(gelu_tanh(j & 1 ? x2[j / 2].y : x2[j / 2].x) * inv);
                    word[j / 4] = (word[j / 4] & ~(0xffu << 8 * (j % 4))) | (uint32_t(max(-128, min(127, code))) & 0xffu) << 8 * (j % 4);
                }
            }
            codes = make_uint2(word[0], word[1]);
        }
        if (first + c * kChunk + lane * 8 < k) *reinterpret_cast<uint2*>(dst + c * kChunk) = codes;
    }
}

// ---- row-wise INT8 (one scale per row), optional exact hi / lo split -----------------------------------------------------
template <bool HILO> WQ_DEVICE void store_row_codes(const float* v, float inv, int8_t* __restrict__ hi, int8_t* __restrict__ lo, int64_t offset) {
    int h[8], l[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float t = v[j] * inv;
        h[j] = __float2int_rn(t);
        if (HILO) l[j] = __float2int_rn((t - float(h[j])) * 254.f);
    }
    *reinterpret_cast<uint2*>(hi + offset) = make_uint2(pack_bytes(h[0], h[1], h[2], h[3]), pack_bytes(h[4], h[5], h[6], h[7]));
    if (HILO) *reinterpret_cast<uint2*>(lo + offset) = make_uint2(pack_bytes(l[0], l[1], l[2], l[3]), pack_bytes(l[4], l[5], l[6], l[7]));
}

// Rows of up to 8192 values: five CTAs per SM (at most 51 registers per thread) -- these kernels are bound by instruction issue and by
// the latency of their two CTA-wide reductions, so resident warps count for more than registers.
template <class T, int GROUP, bool HILO, int ACT, int CPW>
__global__ void __launch_bounds__(kRowThreads, CPW > 0 && CPW <= 4 ? 5 : 1) quantize_rows(const T* __restrict__ x, int8_t* __restrict__ hi, int8_t* __restrict__ lo,
                                                             float* __restrict__ scale, int k, int64_t ldx, const T* __restrict__ act_weight, float eps,
                                                             RowShift shift) {
    __shared__ float sum_slots[9], max_slots[8];
    dependents_may_start();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x;
    const T* src = first_row(x, ldx, shift) + row * ldx;
    float amax = 0.f;
    if constexpr (CPW > 0) {
        float v[CPW][8];
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int col = (warp + 8 * i) * kChunk + lane * 8;
            load_op<T, ACT>(src, k, col, v[i], col < k);
        }
        if constexpr (ACT == kActRms) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < CPW; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
            const float inv_rms = cta_inverse_rms(ss, sum_slots, k, eps);
#pragma unroll
            for (int i = 0; i < CPW; ++i) {
                const int col = (warp + 8 * i) * kChunk + lane * 8;
                scale_by_rms(v[i], inv_rms, act_weight, col, col < k);
            }
        }
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            rotate_chunk<GROUP>(v[i]);
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[i][j]));
        }
        amax = cta_max(amax, max_slots);
        const float inv = amax > 0.f ? 127.f / amax : 0.f;
        if (threadIdx.x == 0) scale[row] = amax * group_norm<GROUP>() / 127.f;
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int col = (warp + 8 * i) * kChunk + lane * 8;
            if (col < k) store_row_codes<HILO>(v[i], inv, hi, lo, row * k + col);
        }
    } else {
        float inv_rms = 1.f;
        if constexpr (ACT == kActRms) {
            float ss = 0.f;
            for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
                float v[8];
                load_eight(src + base + lane * 8, v, base + lane * 8 < k);
#pragma unroll
                for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
            }
            inv_rms = cta_inverse_rms(ss, sum_slots, k, eps);
        }
        for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
            float v[8];
            const bool valid = base + lane * 8 < k;
            load_op<T, ACT>(src, k, base + lane * 8, v, valid);
            if constexpr (ACT == kActRms) scale_by_rms(v, inv_rms, act_weight, base + lane * 8, valid);
            rotate_chunk<GROUP>(v);
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
        }
        amax = cta_max(amax, max_slots);
        const float inv = amax > 0.f ? 127.f / amax : 0.f;
        if (threadIdx.x == 0) scale[row] = amax * group_norm<GROUP>() / 127.f;
        for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
            float v[8];
            const bool valid = base + lane * 8 < k;
            load_op<T, ACT>(src, k, base + lane * 8, v, valid);
            if constexpr (ACT == kActRms) scale_by_rms(v, inv_rms, act_weight, base + lane * 8, valid);
            rotate_chunk<GROUP>(v);
            if (valid) store_row_codes<HILO>(v, inv, hi, lo, row * k + base + lane * 8);
        }
    }
}

// ---- rotated rows, sixteen values a lane ---------------------------------------------------------------------------------------
// A half warp holds a chunk of 256 as sixteen consecutive values a lane: the two low base-4 digits of the index lie inside a lane.  One exchange
// through shared memory turns the chunk over, lane i then holds the elements i + 16 j, and the two high digits lie inside a lane as well.
// (rotate_chunk moves the digits between lanes with 60 shuffles for eight values, one a clock and SM; this takes 20 shared-memory
// instructions for sixteen.)  The additions are those of rotate_chunk, operand by operand, so the codes are the same.
// Measured (one scale a row, groups of 256, alone): 4096 x 3072 22.7 us with the shuffles, 14.4 so (20.5 and 12.6 in a graph); 16384 x 3072 76.6 and 43.9.
// Few rows take longer this way: the rules at launch_blocks() and launch_rows().
constexpr int kTurnStride = 20, kTurnFloats = 16 * kTurnStride + 16;  // rows 80 bytes apart, the halves of a warp 16 banks apart: no conflicts

// one digit of sixteen values whose mirrored partners are STEP apart: out[d] = (in0 + in1) + (in2 + in3) - 2 in[3 - d].  HUGE_VALUES: with
// 2 in[3 - d] rounded first, which makes infinities of what is beyond 2^127, as rotate_chunk does.
template <int STEP, bool HUGE_VALUES> WQ_DEVICE void h4_digit_of_sixteen(float2* v) {
    const float2 minus_two = make_float2(-2.f, -2.f);
    auto less_twice = [&](float2 s, float2 x) {
        if constexpr (HUGE_VALUES) return make_float2(__fadd_rn(s.x, -__fmul_rn(2.f, x.x)), __fadd_rn(s.y, -__fmul_rn(2.f, x.y)));
        return __ffma2_rn(x, minus_two, s);
    };
    if constexpr (STEP == 1) {
#pragma unroll
        for (int g = 0; g < 8; g += 2) {
            const float2 a = v[g], b = v[g + 1];
            const float sum = (a.x + a.y) + (b.x + b.y);
            const float2 s = make_float2(sum, sum);
            v[g] = less_twice(s, make_float2(b.y, b.x));
            v[g + 1] = less_twice(s, make_float2(a.y, a.x));
        }
    } else {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const float2 x0 = v[g], x1 = v[g + 2], x2 = v[g + 4], x3 = v[g + 6];
            const float2 s = __fadd2_rn(__fadd2_rn(x0, x1), __fadd2_rn(x2, x3));
            v[g] = less_twice(s, x3);
            v[g + 2] = less_twice(s, x2);
            v[g + 4] = less_twice(s, x1);
            v[g + 6] = less_twice(s, x0);
        }
    }
}
// v: elements 16 i .. + 15 of the chunk -> for groups of 64 and 256 elements i + 16 j, rotated (`turn`: this half warp's kTurnFloats)
template <int GROUP, bool HUGE_VALUES> WQ_DEVICE void rotate_sixteen(float2* v, float* turn, int i) {
    h4_digit_of_sixteen<1, HUGE_VALUES>(v);
    h4_digit_of_sixteen<4, HUGE_VALUES>(v);
    if constexpr (GROUP > 16) {
        __syncwarp();  // the chunk before this one has been read
#pragma unroll
        for (int j = 0; j < 8; j += 2) *reinterpret_cast<float4*>(turn + i * kTurnStride + 2 * j) = make_float4(v[j].x, v[j].y, v[j + 1].x, v[j + 1].y);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = make_float2(turn[2 * j * kTurnStride + i], turn[(2 * j + 1) * kTurnStride + i]);
        h4_digit_of_sixteen<1, HUGE_VALUES>(v);
        if constexpr (GROUP == 256) h4_digit_of_sixteen<4, HUGE_VALUES>(v);
    }
}
// The rotation keeps the values' root mean square (but for its factor): where no output is as large as this, nothing on the way was.
constexpr float kHuge = 1e38f;
// Sixteen codes, the low bytes of c in the order rotate_sixteen leaves the values in -> the bytes 16 i .. + 15 of the chunk, stored (rows of codes
// need 8-byte alignment only).
template <int GROUP> WQ_DEVICE void store_sixteen(const uint32_t* c, float* turn, int i, int8_t* at, bool valid) {
    uint4 word;
    if constexpr (GROUP == 16) {
        word = make_uint4(low_bytes(c[0], c[1], c[2], c[3]), low_bytes(c[4], c[5], c[6], c[7]), low_bytes(c[8], c[9], c[10], c[11]),
                          low_bytes(c[12], c[13], c[14], c[15]));
    } else {
        uint8_t* bytes = reinterpret_cast<uint8_t*>(turn);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; ++j) bytes[16 * j + i] = uint8_t(c[j]);
        __syncwarp();
        word = *reinterpret_cast<const uint4*>(bytes + 16 * i);
    }
    if (!valid) return;
    if ((reinterpret_cast<uintptr_t>(at) & 15) == 0) {
        *reinterpret_cast<uint4*>(at) = word;
    } else {
        *reinterpret_cast<uint2*>(at) = make_uint2(word.x, word.y);
        *reinterpret_cast<uint2*>(at + 8) = make_uint2(word.z, word.w);
    }
}
template <class T> WQ_DEVICE void load_sixteen(const T* p, float2* v, bool valid) {
    float low[8], high[8];
    load_eight(p, low, valid);
    load_eight(p + 8, high, valid);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = make_float2(low[2 * j], low[2 * j + 1]);
        v[j + 4] = make_float2(high[2 * j], high[2 * j + 1]);
    }
}
// Codes of t = v inv.  PLAIN: every t is a number within 127.5 of zero, so one addition rounds it; else by the conversion, which saturates and
// makes 0 of what is no number.  (Scalar products: the compiler fuses a two-wide one with the addition behind it, __fmul2_rn() and
// mul.rn.f32x2 alike, which puts values next to a tie on the wrong side.)
template <bool PLAIN> WQ_DEVICE void codes_of_sixteen(const float2* v, const float2* inv, uint32_t* codes) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float t = __fmul_rn(j & 1 ? v[j / 2].y : v[j / 2].x, inv[j >> 3].x);
        if constexpr (PLAIN) codes[j] = __float_as_uint(__fadd_rn(t, kRoundMagic));
        else codes[j] = uint32_t(max(-128, min(127, __float2int_rn(t))));
    }
}

template <class T, int GROUP>
__global__ void __launch_bounds__(256) quantize_blocks_rotated(const T* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale, int64_t row0,
                                                               uint32_t items, int k, int64_t ldx, RowShift shift) {
    __shared__ __align__(16) float turns[16 * kTurnFloats];
    dependents_may_start();
    const int i = threadIdx.x & 15, half = threadIdx.x >> 4;
    // an item is a chunk of a row; the items of all rows are numbered through, so that short rows leave no thread idle
    const uint32_t item = blockIdx.x * 16 + half, chunks = uint32_t(k + kChunk - 1) / kChunk;
    if (item - (half & 1) >= items) return;  // both halves of a warp, or none
    float* turn = turns + half * kTurnFloats;
    const int kblocks = (k + kBlockK - 1) / kBlockK, base = int(item % chunks) * kChunk;
    const int64_t row = row0 + item / chunks;
    const int col = base + 16 * i;
    const bool inside = item < items && col < k;
    float2 v[8];
    const T* src = first_row(x, ldx, shift) + row * ldx + col;
    load_sixteen(src, v, inside);
    rotate_sixteen<GROUP, false>(v, turn, i);
    float strict = 0.f;  // absmax, or NaN
#pragma unroll
    for (int j = 0; j < 8; ++j) strict = magnitude_or_nan(strict, magnitude_or_nan(v[j].x, v[j].y));
    const bool ordinary = __all_sync(0xffffffffu, fabsf(strict) < kHuge);
    if (!std::is_same<T, __half>::value && !ordinary) {
        load_sixteen(src, v, inside);
        rotate_sixteen<GROUP, true>(v, turn, i);
    }
    // absmax of the chunk's two blocks: lanes 0-7 end with the first block's, lanes 8-15 with the second's.  (In groups of 16 a lane's values
    // lie in one block, else eight in each.)
    float part[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j) part[j >> 2] = fmaxf(part[j >> 2], fmaxf(fabsf(v[j].x), fabsf(v[j].y)));
    float amax = fmaxf(part[0], part[1]);
    if constexpr (GROUP > 16) amax = fmaxf(i & 8 ? part[1] : part[0], __shfl_xor_sync(0xffffffffu, i & 8 ? part[0] : part[1], 8));
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    const int block = base / kBlockK + (i >> 3);
    const float own_inv = amax > 0.f ? 127.f / amax : 0.f;
    if ((i & 7) == 0 && block < kblocks && item < items) scale[row * kblocks + block] = amax * group_norm<GROUP>() / 127.f;
    float2 inv[2] = {make_float2(own_inv, own_inv), make_float2(own_inv, own_inv)};
    if constexpr (GROUP > 16) {
        const float other = __shfl_xor_sync(0xffffffffu, own_inv, 8);
        inv[i & 8 ? 0 : 1] = make_float2(other, other);
    }
    uint32_t c[16];
    if (ordinary && __all_sync(0xffffffffu, own_inv < kHuge)) codes_of_sixteen<true>(v, inv, c);
    else codes_of_sixteen<false>(v, inv, c);
    store_sixteen<GROUP>(c, turn, i, q + row * k + col, inside);
}

// One scale per row: a CTA per row, CPH chunks a half warp (K <= 4096 CPH), as many warps as the row has work for.
template <class T, int GROUP, bool HILO, int CPH>
__global__ void __launch_bounds__(256) quantize_rows_rotated(const T* __restrict__ x, int8_t* __restrict__ hi, int8_t* __restrict__ lo, float* __restrict__ scale,
                                                             int k, int64_t ldx, RowShift shift) {
    __shared__ __align__(16) float turns[16 * kTurnFloats];
    __shared__ float max_slots[8];
    dependents_may_start();
    const int i = threadIdx.x & 15, half = threadIdx.x >> 4, halves = blockDim.x >> 4;
    float* turn = turns + half * kTurnFloats;
    const int64_t row = blockIdx.x;
    const T* src = first_row(x, ldx, shift) + row * ldx;
    float2 v[CPH][8];
#pragma unroll
    for (int n = 0; n < CPH; ++n) {
        const int col = (half + n * halves) * kChunk + 16 * i;
        load_sixteen(src + col, v[n], col < k);
    }
    float strict = 0.f;  // absmax, or NaN
#pragma unroll
    for (int n = 0; n < CPH; ++n) {
        rotate_sixteen<GROUP, false>(v[n], turn, i);
#pragma unroll
        for (int j = 0; j < 8; ++j) strict = magnitude_or_nan(strict, magnitude_or_nan(v[n][j].x, v[n][j].y));
    }
    float amax = fabsf(strict);
    const bool ordinary = __all_sync(0xffffffffu, amax < kHuge);
    if (!ordinary) {
        amax = 0.f;
#pragma unroll
        for (int n = 0; n < CPH; ++n) {
            if constexpr (!std::is_same<T, __half>::value) {
                const int col = (half + n * halves) * kChunk + 16 * i;
                load_sixteen(src + col, v[n], col < k);
                rotate_sixteen<GROUP, true>(v[n], turn, i);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fmaxf(fabsf(v[n][j].x), fabsf(v[n][j].y)));
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    if ((threadIdx.x & 31) == 0) max_slots[threadIdx.x >> 5] = amax;
    __syncthreads();
    for (int w = 0; w < int(blockDim.x >> 5); ++w) amax = fmaxf(amax, max_slots[w]);
    const float row_inv = amax > 0.f ? 127.f / amax : 0.f;
    if (threadIdx.x == 0) scale[row] = amax * group_norm<GROUP>() / 127.f;
    const float2 inv[2] = {make_float2(row_inv, row_inv), make_float2(row_inv, row_inv)};
    const bool plain = ordinary && row_inv < kHuge;  // (the same in all lanes of a warp)
#pragma unroll
    for (int n = 0; n < CPH; ++n) {
        const int col = (half + n * halves) * kChunk + 16 * i;
        uint32_t h[16], l[16];
        if constexpr (HILO) {  // as store_row_codes
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float t = (j & 1 ? v[n][j / 2].y : v[n][j / 2].x) * row_inv;
                const int code = __float2int_rn(t);
                h[j] = uint32_t(max(-128, min(127, code)));
                l[j] = uint32_t(max(-128, min(127, __float2int_rn((t - float(code)) * 254.f))));
            }
        } else {
            if (plain) codes_of_sixteen<true>(v[n], inv, h);
            else codes_of_sixteen<false>(v[n], inv, h);
        }
        store_sixteen<GROUP>(h, turn, i, hi + row * k + col, col < k);
        if constexpr (HILO) store_sixteen<GROUP>(l, turn, i, lo + row * k + col, col < k);
    }
}

// ---- few-token paths: op(x), rotated, rounded once to T ---------------------------------------------------------------
template <class T, int GROUP, int ACT>
__global__ void __launch_bounds__(kRowThreads) transform_rows(const T* __restrict__ x, T* __restrict__ out, int k, int64_t ldx,
                                                              const T* __restrict__ act_weight, float eps) {
    __shared__ float slots[9];
    dependents_may_start();  // a few-token linear follows: its digit split may be set up while these rows are transformed
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x;
    const T* src = x + row * ldx;
    float inv_rms = 1.f;
    if constexpr (ACT == kActRms) {
        float ss = 0.f;
        for (int base = warp * kChunk; base < k; base += 8 * kChunk) {
            float v[8];
            load_eight(src + base + lane * 8, v, base + lane * 8 < k);
#pragma unroll
            for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
        }
        inv_rms = cta_inverse_rms(ss, slots, k, eps);
    }
    constexpr float norm = group_norm<GROUP>();
    // gridDim.y CTAs share a row when no row statistic is needed: with one or a few rows every warp then has one chunk and one trip to
    // memory instead of a chain of them
    for (int base = (blockIdx.y * 8 + warp) * kChunk; base < k; base += gridDim.y * 8 * kChunk) {
        float v[8];
        const bool valid = base + lane * 8 < k;
        load_op<T, ACT>(src, k, base + lane * 8, v, valid);
        if constexpr (ACT == kActRms) scale_by_rms(v, inv_rms, act_weight, base + lane * 8, valid);
        rotate_chunk<GROUP>(v);
        if (valid) {
            uint4 packed;
            packed.x = pack_pair<T>(v[0] * norm, v[1] * norm);
            packed.y = pack_pair<T>(v[2] * norm, v[3] * norm);
            packed.z = pack_pair<T>(v[4] * norm, v[5] * norm);
            packed.w = pack_pair<T>(v[6] * norm, v[7] * norm);
            *reinterpret_cast<uint4*>(out + row * k + base + lane * 8) = packed;
        }
    }
}

// Standalone rotation (a warp per 256-element chunk, persistent): out = T(rotated * 1 / sqrt(GROUP)).
template <class T, int GROUP>
__global__ void __launch_bounds__(256) rotate_groups(const T* __restrict__ x, T* __restrict__ out, int m, int k, int64_t ldx) {
    const int lane = threadIdx.x & 31;
    const int chunks = (k + kChunk - 1) / kChunk;
    const int64_t items = int64_t(m) * chunks, stride = int64_t(gridDim.x) * 8;
    constexpr float norm = group_norm<GROUP>();
    for (int64_t item = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5); item < items; item += stride) {
        const int64_t row = item / chunks;
        const int col = int(item % chunks) * kChunk + lane * 8;
        float v[8];
        load_eight(x + row * ldx + col, v, col < k);
        rotate_chunk<GROUP>(v);
        if (col < k) {
            uint4 packed;
            packed.x = pack_pair<T>(v[0] * norm, v[1] * norm);
            packed.y = pack_pair<T>(v[2] * norm, v[3] * norm);
            packed.z = pack_pair<T>(v[4] * norm, v[5] * norm);
            packed.w = pack_pair<T>(v[6] * norm, v[7] * norm);
            *reinterpret_cast<uint4*>(out + row * k + col) = packed;
        }
    }
}

// ---- host dispatch ----------------------------------------------------------------------------------------------------
static int device_sm_count() {
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;
}

static int persistent_ctas(int64_t warps_of_work) {
    const int64_t ctas = (warps_of_work + 7) / 8, cap = int64_t(device_sm_count()) * 8;  // 8 CTAs of 256 threads fill an SM
    return int(ctas < cap ? (ctas < 1 ? 1 : ctas) : cap);
}

// A rotation without an input operation: whether the kernel with sixteen values a lane is the faster one.  It needs fewer instructions, but takes longer
// for one chunk (the turn through shared memory), so where few chunks or rows fill no more than a wave, the kernel with eight values a lane and shuffles
// stays.  Both measured over K of 512 to 16384 and 1 to 8192 rows, BF16 and FP32, device time in a graph (shuffles and this, us; BF16): blocks
// of 64, 16 x 5120 1.87 and 2.21 | 128 x 5120 2.43 and 2.55 | 256 x 5120 3.50 and 3.27 | 8192 x 5120 47.7 and 36.0; 8192 x 1024 11.8 and 9.4;
// rows in groups of 64, 16 x 2048 1.85 and 2.05 | 512 x 2048 2.83 and 2.71 | 16 x 9216 3.36 and 3.07.  hi and lo in groups of 64: 512 x 5120 6.43
// and 5.78, but where the other kernel's eight warps have the same number of chunks it is faster, 1024 x 8192 10.7 and 11.4, and so it is on long
// rows while they are few, 256 x 13824 6.9 and 7.8.  hi and lo in groups of 16: two more digits' worth of registers for twelve shuffles, 1560 x 13824
// 19.9 and 25.0.  FP32, twice the bytes: rows in groups of 64, 8192 x 8192 63.8 and 72.6 | 8192 x 9216 121.8 and 89.8 | 2048 x 1536 6.4 and 6.9.
template <class T, int GROUP> static bool sixteen_values_win_blocks(int64_t chunks_of_all_rows) {
    constexpr int kChunksOfAnSm = sizeof(T) == 4 ? (GROUP == 16 ? 60 : GROUP == 64 ? 120 : 24) : GROUP == 256 ? 10 : 22;
    return chunks_of_all_rows >= kChunksOfAnSm * device_sm_count();
}
template <class T, int GROUP, bool HILO> static bool sixteen_values_win_rows(int m, int k) {
    if (k > 16384) return false;  // (more than a CTA's registers hold)
    constexpr bool kWide = sizeof(T) == 4;
    const bool even = (k + kChunk - 1) / kChunk % 8 == 0;
    if (GROUP == 256) return (m > 128 || k > (HILO ? 4096 : 2048)) && !(kWide && HILO && even && m < 4096);
    if (!HILO && !kWide) return m > 256 || k > 4096;
    return !even && !(kWide && k > 1024 && k <= 2048) && m >= (!HILO ? 257 : k <= 12288 ? 512 : 2048);
}

template <class T, int GROUP, int ACT>
static int launch_blocks(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, const void* act_weight, float eps, const RowShift& shift,
                         cudaStream_t stream) {
    auto src = static_cast<const T*>(x);
    auto aw = static_cast<const T*>(act_weight);
    if constexpr (ACT == kActRms) {
        if (k <= 2048) quantize_blocks_rms<T, GROUP, 1><<<m, kRowThreads, 0, stream>>>(src, q, scale, m, k, ldx, aw, eps, shift);
        else if (k <= 4096) quantize_blocks_rms<T, GROUP, 2><<<m, kRowThreads, 0, stream>>>(src, q, scale, m, k, ldx, aw, eps, shift);
        else if (k <= 8192) quantize_blocks_rms<T, GROUP, 4><<<m, kRowThreads, 0, stream>>>(src, q, scale, m, k, ldx, aw, eps, shift);
        else if (k <= 16384) quantize_blocks_rms<T, GROUP, 8><<<m, kRowThreads, 0, stream>>>(src, q, scale, m, k, ldx, aw, eps, shift);
        else quantize_blocks_rms<T, GROUP, 0><<<m, kRowThreads, 0, stream>>>(src, q, scale, m, k, ldx, aw, eps, shift);
    } else {
        const int chunks = (k + kChunk - 1) / kChunk;
        if constexpr (ACT == kActGelu && GROUP == 0) {  // (a rotation needs every accurate value)
            // Four chunks a warp want enough warps: 20 an SM (BF16, one chunk a warp with tanhf and this, us: 256 rows of 5888 values 4.0 and 4.5,
            // 512 of 6144 6.2 and 6.1, 1024 of 6144 10.0 and 8.4, 256 of 13824 6.8 and 6.7).
            const int64_t groups = (chunks + kGeluChunks - 1) / kGeluChunks;
            if (m * groups >= 20 * device_sm_count()) {
                const int64_t most = (int64_t(1) << 30) / groups;
                for (int64_t row0 = 0; row0 < m; row0 += most) {
                    const uint32_t items = uint32_t((m - row0 < most ? m - row0 : most) * groups);
                    quantize_blocks_gelu<T><<<(items + 7) / 8, 256, 0, stream>>>(src, q, scale, row0, items, k, ldx, shift);
                }
                return int(cudaGetLastError());
            }
        }
        if constexpr (GROUP > 0 && ACT == kActNone) {
            if (sixteen_values_win_blocks<T, GROUP>(int64_t(m) * chunks)) {
                const int64_t most = (int64_t(1) << 30) / chunks;
                for (int64_t row0 = 0; row0 < m; row0 += most) {
                    const uint32_t items = uint32_t((m - row0 < most ? m - row0 : most) * chunks);
                    quantize_blocks_rotated<T, GROUP><<<(items + 15) / 16, 256, 0, stream>>>(src, q, scale, row0, items, k, ldx, shift);
                }
                return int(cudaGetLastError());
            }
        }
        for (int64_t row0 = 0; row0 < m; row0 += 65535) {
            const dim3 grid((chunks + 7) / 8, unsigned(m - row0 < 65535 ? m - row0 : 65535));
            quantize_blocks_items<T, GROUP, ACT><<<grid, 256, 0, stream>>>(src, q, scale, row0, k, ldx, shift);
        }
    }
    return int(cudaGetLastError());
}

template <class T, int ACT>
static int blocks_by_group(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, int group, const void* aw, float eps, const RowShift& shift,
                           cudaStream_t stream) {
    switch (group) {
        case 0: return launch_blocks<T, 0, ACT>(x, q, scale, m, k, ldx, aw, eps, shift, stream);
        case 16: return launch_blocks<T, 16, ACT>(x, q, scale, m, k, ldx, aw, eps, shift, stream);
        case 64: return launch_blocks<T, 64, ACT>(x, q, scale, m, k, ldx, aw, eps, shift, stream);
        case 256: return launch_blocks<T, 256, ACT>(x, q, scale, m, k, ldx, aw, eps, shift, stream);
    }
    return -1;
}

template <class T>
static int blocks_by_act(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, int group, int act, const void* aw, float eps,
                         const RowShift& shift, cudaStream_t stream) {
    switch (act) {
        case kActNone: return blocks_by_group<T, kActNone>(x, q, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActRms: return blocks_by_group<T, kActRms>(x, q, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActSwiglu: return blocks_by_group<T, kActSwiglu>(x, q, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActGelu: return blocks_by_group<T, kActGelu>(x, q, scale, m, k, ldx, group, aw, eps, shift, stream);
    }
    return -1;
}

template <class T, int GROUP, bool HILO, int ACT>
static int launch_rows(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, const void* act_weight, float eps,
                       const RowShift& shift, cudaStream_t stream) {
    auto src = static_cast<const T*>(x);
    auto aw = static_cast<const T*>(act_weight);
    // (rms_norm: the order of the row's sum is that of eight values a lane; gelu and swiglu: how their last product and the rotation's first sum
    // are fused is that kernel's)
    if constexpr (GROUP > 0 && ACT == kActNone && !(GROUP == 16 && HILO)) {
        if (sixteen_values_win_rows<T, GROUP, HILO>(m, k)) {
            const int chunks = (k + kChunk - 1) / kChunk, per_half = k <= 4096 ? 1 : k <= 8192 ? 2 : 4;
            const int threads = 32 * ((chunks + 2 * per_half - 1) / (2 * per_half));
            if (per_half == 1) quantize_rows_rotated<T, GROUP, HILO, 1><<<m, threads, 0, stream>>>(src, hi, lo, scale, k, ldx, shift);
            else if (per_half == 2) quantize_rows_rotated<T, GROUP, HILO, 2><<<m, threads, 0, stream>>>(src, hi, lo, scale, k, ldx, shift);
            else quantize_rows_rotated<T, GROUP, HILO, 4><<<m, threads, 0, stream>>>(src, hi, lo, scale, k, ldx, shift);
            return int(cudaGetLastError());
        }
    }
    auto kernel = quantize_rows<T, GROUP, HILO, ACT, 0>;
    if (k <= 2048) kernel = quantize_rows<T, GROUP, HILO, ACT, 1>;
    else if (k <= 4096) kernel = quantize_rows<T, GROUP, HILO, ACT, 2>;
    else if (k <= 8192) kernel = quantize_rows<T, GROUP, HILO, ACT, 4>;
    else if (k <= 16384) kernel = quantize_rows<T, GROUP, HILO, ACT, 8>;
    kernel<<<m, kRowThreads, 0, stream>>>(src, hi, lo, scale, k, ldx, aw, eps, shift);
    return int(cudaGetLastError());
}

template <class T, bool HILO, int ACT>
static int rows_by_group(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, int group, const void* aw, float eps,
                         const RowShift& shift, cudaStream_t stream) {
    switch (group) {
        case 0: return launch_rows<T, 0, HILO, ACT>(x, hi, lo, scale, m, k, ldx, aw, eps, shift, stream);
        case 16: return launch_rows<T, 16, HILO, ACT>(x, hi, lo, scale, m, k, ldx, aw, eps, shift, stream);
        case 64: return launch_rows<T, 64, HILO, ACT>(x, hi, lo, scale, m, k, ldx, aw, eps, shift, stream);
        case 256: return launch_rows<T, 256, HILO, ACT>(x, hi, lo, scale, m, k, ldx, aw, eps, shift, stream);
    }
    return -1;
}

template <class T, bool HILO>
static int rows_by_act(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, int group, int act, const void* aw, float eps,
                       const RowShift& shift, cudaStream_t stream) {
    switch (act) {
        case kActNone: return rows_by_group<T, HILO, kActNone>(x, hi, lo, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActRms: return rows_by_group<T, HILO, kActRms>(x, hi, lo, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActSwiglu: return rows_by_group<T, HILO, kActSwiglu>(x, hi, lo, scale, m, k, ldx, group, aw, eps, shift, stream);
        case kActGelu: return rows_by_group<T, HILO, kActGelu>(x, hi, lo, scale, m, k, ldx, group, aw, eps, shift, stream);
    }
    return -1;
}

template <class T, int GROUP>
static int launch_transform(const void* x, void* out, int m, int k, int64_t ldx, int act, const void* act_weight, float eps, cudaStream_t stream) {
    auto src = static_cast<const T*>(x);
    auto aw = static_cast<const T*>(act_weight);
    auto dst = static_cast<T*>(out);
    // few rows: the CTAs of a row take its chunks in turn (not with rms_norm, whose row sum is formed inside one CTA)
    const int chunk_groups = (k + 8 * kChunk - 1) / (8 * kChunk);
    const dim3 grid(m, m < 64 ? (chunk_groups < 64 ? chunk_groups : 64) : 1);
    switch (act) {
        case kActNone: transform_rows<T, GROUP, kActNone><<<grid, kRowThreads, 0, stream>>>(src, dst, k, ldx, aw, eps); break;
        case kActRms: transform_rows<T, GROUP, kActRms><<<m, kRowThreads, 0, stream>>>(src, dst, k, ldx, aw, eps); break;
        case kActSwiglu: transform_rows<T, GROUP, kActSwiglu><<<grid, kRowThreads, 0, stream>>>(src, dst, k, ldx, aw, eps); break;
        case kActGelu: transform_rows<T, GROUP, kActGelu><<<grid, kRowThreads, 0, stream>>>(src, dst, k, ldx, aw, eps); break;
        default: return -1;
    }
    return int(cudaGetLastError());
}

template <class T>
static int transform_by_group(const void* x, void* out, int m, int k, int64_t ldx, int group, int act, const void* aw, float eps, cudaStream_t stream) {
    switch (group) {
        case 0: return launch_transform<T, 0>(x, out, m, k, ldx, act, aw, eps, stream);
        case 16: return launch_transform<T, 16>(x, out, m, k, ldx, act, aw, eps, stream);
        case 64: return launch_transform<T, 64>(x, out, m, k, ldx, act, aw, eps, stream);
        case 256: return launch_transform<T, 256>(x, out, m, k, ldx, act, aw, eps, stream);
    }
    return -1;
}

template <class T>
static int rotate_by_group(const void* x, void* out, int m, int k, int64_t ldx, int group, cudaStream_t stream) {
    auto src = static_cast<const T*>(x);
    auto dst = static_cast<T*>(out);
    const int ctas = persistent_ctas(int64_t(m) * ((k + kChunk - 1) / kChunk));
    if (group == 16) rotate_groups<T, 16><<<ctas, 256, 0, stream>>>(src, dst, m, k, ldx);
    else if (group == 64) rotate_groups<T, 64><<<ctas, 256, 0, stream>>>(src, dst, m, k, ldx);
    else if (group == 256) rotate_groups<T, 256><<<ctas, 256, 0, stream>>>(src, dst, m, k, ldx);
    else return -1;
    return int(cudaGetLastError());
}

}  // namespace wq

using namespace wq;

static int quantize_blocks_entry(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                                 const void* act_weight, float eps, const RowShift& shift, cudaStream_t stream) {
    if (m <= 0) return 0;
    if (k <= 0 || k % 8 || (group && k % group)) return -2;
    if (dtype == 0) return blocks_by_act<__half>(x, q, scale, m, k, ldx, group, act, act_weight, eps, shift, stream);
    if (dtype == 1) return blocks_by_act<bf16>(x, q, scale, m, k, ldx, group, act, act_weight, eps, shift, stream);
    if (dtype != 2 || act) return -1;
    return blocks_by_group<float, kActNone>(x, q, scale, m, k, ldx, group, nullptr, 0.f, shift, stream);
}

static int quantize_entry(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                          const void* act_weight, float eps, const RowShift& shift, cudaStream_t stream) {
    if (m <= 0) return 0;
    if (k <= 0 || k % 8 || (group && k % group)) return -2;
    if (dtype == 0)
        return lo ? rows_by_act<__half, true>(x, hi, lo, scale, m, k, ldx, group, act, act_weight, eps, shift, stream)
                  : rows_by_act<__half, false>(x, hi, lo, scale, m, k, ldx, group, act, act_weight, eps, shift, stream);
    if (dtype == 1)
        return lo ? rows_by_act<bf16, true>(x, hi, lo, scale, m, k, ldx, group, act, act_weight, eps, shift, stream)
                  : rows_by_act<bf16, false>(x, hi, lo, scale, m, k, ldx, group, act, act_weight, eps, shift, stream);
    if (dtype != 2 || act) return -1;
    return lo ? rows_by_group<float, true, kActNone>(x, hi, lo, scale, m, k, ldx, group, nullptr, 0.f, shift, stream)
              : rows_by_group<float, false, kActNone>(x, hi, lo, scale, m, k, ldx, group, nullptr, 0.f, shift, stream);
}

WQ_API int wq8_quantize_blocks(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                               const void* act_weight, float eps, float* /*inv_rms: rows of any K are handled inside one kernel*/, cudaStream_t stream) {
    return quantize_blocks_entry(x, q, scale, m, k, ldx, dtype, group, act, act_weight, eps, RowShift{nullptr, 0, 0}, stream);
}

// wq8_quantize_blocks reading rows first + counter[0] * step ... of x (the outputs start at row 0): counter on the GPU, read at run time.
WQ_API int wq8_quantize_blocks_at(const void* x, int8_t* q, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                                  const void* act_weight, float eps, float* /*inv_rms*/, const long long* counter, long long first, long long step,
                                  cudaStream_t stream) {
    return quantize_blocks_entry(x, q, scale, m, k, ldx, dtype, group, act, act_weight, eps, RowShift{counter, first, step}, stream);
}

WQ_API int wq8_quantize(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                        const void* act_weight, float eps, cudaStream_t stream) {
    return quantize_entry(x, hi, lo, scale, m, k, ldx, dtype, group, act, act_weight, eps, RowShift{nullptr, 0, 0}, stream);
}

// wq8_quantize reading rows first + counter[0] * step ... of x: counter on the GPU, read at run time.
WQ_API int wq8_quantize_at(const void* x, int8_t* hi, int8_t* lo, float* scale, int m, int k, int64_t ldx, int dtype, int group, int act,
                           const void* act_weight, float eps, const long long* counter, long long first, long long step, cudaStream_t stream) {
    return quantize_entry(x, hi, lo, scale, m, k, ldx, dtype, group, act, act_weight, eps, RowShift{counter, first, step}, stream);
}

WQ_API int wq8_transform_rows(const void* x, void* out, int m, int k, int64_t ldx, int dtype, int group, int act, const void* act_weight, float eps,
                              cudaStream_t stream) {
    if (m <= 0) return 0;
    if (k <= 0 || k % 8 || (group && k % group)) return -2;
    if (dtype == 0) return transform_by_group<__half>(x, out, m, k, ldx, group, act, act_weight, eps, stream);
    if (dtype == 1) return transform_by_group<bf16>(x, out, m, k, ldx, group, act, act_weight, eps, stream);
    return -1;
}

WQ_API int wq8_rotate_groups(const void* x, void* out, int m, int k, int64_t ldx, int dtype, int group, cudaStream_t stream) {
    if (m <= 0) return 0;
    if (k <= 0 || k % 8 || (group && k % group)) return -2;
    if (dtype == 0) return rotate_by_group<__half>(x, out, m, k, ldx, group, stream);
    if (dtype == 1) return rotate_by_group<bf16>(x, out, m, k, ldx, group, stream);
    return -1;
}
