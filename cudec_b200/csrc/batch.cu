// C-ABI batch entries for the byte-oriented LZ formats (LZ4, raw Snappy):
// the CTA-per-chunk decoder (lz_cta_kernel.cuh), persistent over the batch.
//
// Contract (include/cudec.h): synchronous validation with no CUDA call on a
// reject, then the pending CUDA error is consumed, the kernel is submitted on
// the caller's stream, and the submission status is returned. Replaces
// iderex/cudec src/batch.cu:6-31 with validate_batch_args at
// src/lz4_decode.cuh:187-201 and the limit at src/batch_limits.h:28.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "cudec.h"
#include "launch.h"
#include "lz_cta_kernel.cuh"

namespace cdb {

cudec_status validate_batch(const void* const* src, const size_t* src_sizes,
                            void* const* dst, const size_t* caps, size_t n,
                            const cudec_chunk_result* results) {
    if (src == nullptr || src_sizes == nullptr || dst == nullptr ||
        caps == nullptr || results == nullptr ||
        reinterpret_cast<uintptr_t>(results) % 16 != 0 || n == 0 ||
        n > kMaxBatchChunks) {
        return CUDEC_ERR_INVALID_ARGUMENT;
    }
    return CUDEC_OK;
}

namespace {

constexpr int kMaxDevices = 64;
std::atomic<int> g_sm_count[kMaxDevices];

// Chunks per SM up to which a batch's chunks get 512 or 256 threads each. Us
// per batch of 64 KiB chunks with 512 / 256 / 128 threads on 148 SMs (128: with
// the wide kernel beside, which finds nothing): LZ4 74 chunks 129 / 166 / 275,
// 148 131 / 168 / 275, 200 221 / 191 / 284, 296 244 / 191 / 287, 370 326 / 214 /
// 311, 444 347 / 214 / 311, 518 426 / 330 / 317, 592 453 / 363 / 331, 1,036 770 /
// 521 / 412; Snappy 148 146 / 189 / 290, 296 265 / 209 / 315, 444 379 / 231 /
// 327, 592 490 / 381 / 340; 16 LZ4 chunks of 4 MiB 5,706 / 7,993 / 8,186.
constexpr size_t kWideMax = 1, kMediumMax = 3;
// Threads of the wide CTAs beside narrow ones. 512 are quicker where the largest
// chunk ends the batch (8,000 uneven Snappy chunks 2,869 us instead of 4,228,
// 2,000 1,551 and 2,259, 30,000 uneven LZ4 chunks 3,610 and 3,698; 1,024 alike
// 412 and 412), and not measured yet over other sizes.
constexpr uint32_t kWideThreads = 256;
// Up to here the wide CTAs read every capacity each (148 x 1 MiB out of L2), and
// the narrow ones of large chunks some of them (is_large). 100,000 LZ4 pages of
// 4 KiB take 3,610 us; with 1,000, 50,000 or all of them in slots of 256 KiB
// 3,656, 3,743 and 3,784.
constexpr size_t kWideBeside = 1 << 17;

}  // namespace

int device_sm_count(int dev) {
    if (dev < 0 || dev >= kMaxDevices) return 0;
    int v = g_sm_count[dev].load(std::memory_order_relaxed);
    if (v > 0) return v;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
        return 0;
    g_sm_count[dev].store(v, std::memory_order_relaxed);
    return v;
}

// The kernels' shared state is 29 KB with 128 threads, 56 KB with 256 and 111 KB
// with 512. Above 48 KB it is opted into, once per device, format and width (the
// narrow one's opt-in changes nothing).
template <class F, uint32_t T>
cudaError_t prepare_cta(int dev) {
    static std::atomic<bool> ready[kMaxDevices];
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (ready[dev].load(std::memory_order_acquire)) return cudaSuccess;
    constexpr int kSmem = static_cast<int>(sizeof(lzc::Shm<F, T>));
    cudaError_t e = cudaFuncSetAttribute(lzc::lz_cta_kernel<F, T>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if constexpr (T == kWideThreads)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(lzc::lz_wide_kernel<F, T>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e == cudaSuccess) ready[dev].store(true, std::memory_order_release);
    return e;
}

struct Batch {
    const void* const* src;
    const size_t* src_sizes;
    void* const* dst;
    const size_t* caps;
    size_t n;
    cudec_chunk_result* results;
    cudaStream_t stream;
    int dev;
};

// One CTA of T threads per chunk (the hardware hands CTAs out as SMs fall
// free, so uneven chunks balance).
template <class F, uint32_t T>
cudec_status launch_width(const Batch& b) {
    if (prepare_cta<F, T>(b.dev) != cudaSuccess) return CUDEC_ERR_CUDA;
    constexpr size_t kMaxGrid = INT32_MAX;
    const unsigned grid = static_cast<unsigned>(b.n < kMaxGrid ? b.n : kMaxGrid);
    lzc::lz_cta_kernel<F, T><<<grid, T, sizeof(lzc::Shm<F, T>), b.stream>>>(
        b.src, b.src_sizes, b.dst, b.caps, b.n, b.results, 0);
    return cudaGetLastError() == cudaSuccess ? CUDEC_OK : CUDEC_ERR_CUDA;
}

// Many chunks: narrow CTAs, and beside them a wide CTA per SM for the few
// that are large (lz_wide_kernel). The narrow kernel is a programmatic
// dependent of the wide one, which lets it start at once.
template <class F>
cudec_status launch_many(const Batch& b, unsigned sms) {
    if (prepare_cta<F, 128>(b.dev) != cudaSuccess ||
        prepare_cta<F, kWideThreads>(b.dev) != cudaSuccess)
        return CUDEC_ERR_CUDA;
    lzc::lz_wide_kernel<F, kWideThreads>
        <<<sms, kWideThreads, sizeof(lzc::Shm<F, kWideThreads>), b.stream>>>(
            b.src, b.src_sizes, b.dst, b.caps, b.n, b.results);
    if (cudaGetLastError() != cudaSuccess) return CUDEC_ERR_CUDA;
    constexpr size_t kMaxGrid = INT32_MAX;
    cudaLaunchAttribute beside{};
    beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    beside.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(b.n < kMaxGrid ? b.n : kMaxGrid));
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = sizeof(lzc::Shm<F, 128>);
    cfg.stream = b.stream;
    cfg.attrs = &beside;
    cfg.numAttrs = 1;
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, lzc::lz_cta_kernel<F, 128>, b.src, b.src_sizes, b.dst, b.caps,
                           b.n, b.results, static_cast<uint32_t>(sms));
    return e == cudaSuccess ? CUDEC_OK : CUDEC_ERR_CUDA;
}

template <class F>
cudec_status launch_lz_cta(const void* const* src, const size_t* src_sizes, void* const* dst,
                           const size_t* caps, size_t n, cudec_chunk_result* results,
                           cudaStream_t stream) {
    const cudec_status v = validate_batch(src, src_sizes, dst, caps, n, results);
    if (v != CUDEC_OK) return v;
    (void)cudaGetLastError();
    Batch b{src, src_sizes, dst, caps, n, results, stream, 0};
    if (cudaGetDevice(&b.dev) != cudaSuccess) return CUDEC_ERR_CUDA;
    const size_t sms = static_cast<size_t>(device_sm_count(b.dev));
    if (sms == 0) return CUDEC_ERR_CUDA;
    // A wide CTA shortens a chunk's own time, narrow ones use the SM better:
    // wide while the batch leaves SMs idle otherwise.
    if (n <= kWideMax * sms) return launch_width<F, 512>(b);
    if (n <= kMediumMax * sms) return launch_width<F, 256>(b);
    if (n <= kWideBeside) return launch_many<F>(b, static_cast<unsigned>(sms));
    return launch_width<F, 128>(b);
}

}  // namespace cdb

extern "C" {

cudec_status cudec_lz4_decompress_batch(const void* const* d_src_ptrs,
                                        const size_t* d_src_sizes,
                                        void* const* d_dst_ptrs,
                                        const size_t* d_dst_capacities,
                                        size_t chunk_count,
                                        cudec_chunk_result* d_results,
                                        cudec_stream_t stream) {
    return cdb::launch_lz_cta<cdb::lzc::Lz4F>(
        d_src_ptrs, d_src_sizes, d_dst_ptrs, d_dst_capacities,
        chunk_count, d_results, reinterpret_cast<cudaStream_t>(stream));
}

cudec_status cudec_snappy_decompress_batch(const void* const* d_src_ptrs,
                                           const size_t* d_src_sizes,
                                           void* const* d_dst_ptrs,
                                           const size_t* d_dst_capacities,
                                           size_t chunk_count,
                                           cudec_chunk_result* d_results,
                                           cudec_stream_t stream) {
    return cdb::launch_lz_cta<cdb::lzc::SnappyF>(
        d_src_ptrs, d_src_sizes, d_dst_ptrs,
        d_dst_capacities, chunk_count, d_results,
        reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"

#ifdef CDB_PHASE_TIMING
// Profiling builds only: the CTA decoder's phase cycles [0, 16) and event
// counts [16, 32) since the last call (then reset).
extern "C" int cudec_lzc_phase_counters(unsigned long long* out) {
    if (cudaMemcpyFromSymbol(out, cdb::lzc::lzc_cycles, 16 * sizeof(unsigned long long)) !=
            cudaSuccess ||
        cudaMemcpyFromSymbol(out + 16, cdb::lzc::lzc_events, 16 * sizeof(unsigned long long)) !=
            cudaSuccess)
        return 1;
    static const unsigned long long zero[16] = {};
    if (cudaMemcpyToSymbol(cdb::lzc::lzc_cycles, zero, sizeof(zero)) != cudaSuccess ||
        cudaMemcpyToSymbol(cdb::lzc::lzc_events, zero, sizeof(zero)) != cudaSuccess)
        return 1;
    return 0;
}
#endif
