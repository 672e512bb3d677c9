// ABI identification and the cold-cache helper of the tuner.
#include "common.cuh"

namespace wq {

// Reads a buffer twice the size of L2 so that the next launch streams its operands from HBM, as a layer of a model does.
__global__ void __launch_bounds__(256) l2_flush_read(const int4* __restrict__ p, int64_t count, int* sink) {
    int4 acc = make_int4(0, 0, 0, 0);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x) {
        const int4 v = __ldcg(p + i);
        acc.x ^= v.x; acc.y ^= v.y; acc.z ^= v.z; acc.w ^= v.w;
    }
    if ((acc.x ^ acc.y ^ acc.z ^ acc.w) == 0x1f2e3d4c && sink) *sink = 1;  // keeps the loads alive; never true for the zeroed buffer
}

static void* flush_buffer = nullptr;
static int64_t flush_bytes = 0;
static int flush_device = -1;

}  // namespace wq

using namespace wq;

WQ_API int wq8_abi() { return 11; }
WQ_API int wq8_features() { return 1; }

// The buffer comes from cudaMalloc, not from the caller's allocator: tuning during the eager warm-up of a CUDA graph must leave nothing
// in the graph's memory pool.
WQ_API int wq8_l2_flush(int device, int64_t bytes, cudaStream_t stream) {
    if (bytes <= 0) return 0;
    if (flush_bytes < bytes || flush_device != device) {
        int current = 0;
        cudaGetDevice(&current);
        if (current != device) (void)cudaSetDevice(device);
        if (flush_buffer) (void)cudaFree(flush_buffer);
        flush_buffer = nullptr;
        flush_bytes = 0;
        const cudaError_t e = cudaMalloc(&flush_buffer, size_t(bytes) + 16);
        if (e == cudaSuccess) (void)cudaMemset(flush_buffer, 0, size_t(bytes) + 16);
        if (current != device) (void)cudaSetDevice(current);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            flush_buffer = nullptr;
            return 1;
        }
        flush_bytes = bytes;
        flush_device = device;
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    l2_flush_read<<<sms * 8, 256, 0, stream>>>(static_cast<const int4*>(flush_buffer), bytes / 16, static_cast<int*>(flush_buffer) + bytes / 4);
    return int(cudaGetLastError());
}

WQ_API void wq8_l2_flush_release() {
    if (flush_buffer) (void)cudaFree(flush_buffer);
    flush_buffer = nullptr;
    flush_bytes = 0;
    flush_device = -1;
}

// ---- a whole linear in one call ------------------------------------------------------------------------------------
// The quantizer and the GEMM of a row band behind one entry point: a host in an interpreted language otherwise spends more on the two calls, the
// codes' and scales' own allocations and the objects around them than a small linear takes on the GPU.
extern "C" {
int wq8_quantize_blocks(const void*, int8_t*, float*, int, int, int64_t, int, int, int, const void*, float, float*, cudaStream_t);
int wq8_quantize(const void*, int8_t*, int8_t*, float*, int, int, int64_t, int, int, int, const void*, float, cudaStream_t);
int wq8_gemm(const int8_t*, const int8_t*, const float*, const int8_t*, const float*, const void*, const void*, const void*, void*, int, int, int, int, int,
             int, int, int*, int*, cudaStream_t);
void wq8_gemm_workspace(int, int, int, int, int, int, int64_t*);
}

namespace wq {
int path_and_variant(int path, int variant);  // gemm_tc.cu
struct LinearScratch { int64_t codes, low, scales, workspace, total; };  // offsets of the parts, 256-byte aligned
static LinearScratch linear_scratch(int m, int n, int k, int path, int variant, int sms) {
    auto padded = [](int64_t bytes) { return (bytes + 255) / 256 * 256; };
    LinearScratch s{};
    s.low = padded(int64_t(m) * k);
    s.scales = s.low + (path == 1 ? padded(int64_t(m) * k) : 0);
    s.workspace = s.scales + padded(int64_t(m) * (path == 0 ? (k + kBlockK - 1) / kBlockK : 1) * 4);
    int64_t sizes[2];
    wq8_gemm_workspace(m, n, k, variant, sms, 0, sizes);
    s.total = s.workspace + padded(sizes[0]);
    return s;
}
}  // namespace wq

WQ_API int64_t wq8_linear_scratch(int m, int n, int k, int path, int variant, int sms) {
    if (m <= 0 || n <= 0 || k <= 0 || wq::path_and_variant(path, variant)) return 0;
    return wq::linear_scratch(m, n, k, path, variant, sms).total;
}

WQ_API int wq8_linear(const void* x, int64_t ldx, const int8_t* w, const float* sw, const void* bias, const void* residual, const void* rscale, void* y,
                      int m, int n, int k, int dtype, int group, int act, const void* act_weight, float eps, int path, int variant, int sms,
                      void* scratch, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (dtype != 0 && dtype != 1) return -1;
    if (const int code = wq::path_and_variant(path, variant)) return code;
    if (k <= 0 || k % 16 || !scratch || (reinterpret_cast<uintptr_t>(scratch) & 255)) return -2;
    const wq::LinearScratch s = wq::linear_scratch(m, n, k, path, variant, sms);
    auto base = static_cast<int8_t*>(scratch);
    int8_t* low = path == 1 ? base + s.low : nullptr;
    auto scales = reinterpret_cast<float*>(base + s.scales);
    const int code = path == 0 ? wq8_quantize_blocks(x, base, scales, m, k, ldx, dtype, group, act, act_weight, eps, nullptr, stream)
                               : wq8_quantize(x, base, low, scales, m, k, ldx, dtype, group, act, act_weight, eps, stream);
    if (code) return code;
    return wq8_gemm(base, low, scales, w, sw, bias, residual, rscale, y, m, n, k, dtype, variant, sms, 0, reinterpret_cast<int*>(base + s.workspace), nullptr,
                    stream);
}
