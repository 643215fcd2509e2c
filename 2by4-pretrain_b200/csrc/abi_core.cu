// Library-wide pieces of the C ABI: error strings, version, device check.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "sp24_common.cuh"

namespace sp24 {

int check_device() {
    // The answer is cached per device ordinal; concurrent first calls write the same value.
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return runtime_error();
    if (dev >= 0 && dev < 64)
        if (const int known = cached[dev]) return known == 1 ? SP24_OK : SP24_ERR_DEVICE;
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return runtime_error();
    const int ok = major == 10;
    if (dev >= 0 && dev < 64) cached[dev] = ok ? 1 : 2;
    return ok ? SP24_OK : SP24_ERR_DEVICE;
}

// Number of SMs of the current device (cached per device ordinal; 148 if the query fails).
int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        runtime_error();
        return 148;
    }
    if (dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) runtime_error();
        if (n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

int launch_status() {
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return SP24_OK;
    if (getenv("SP24_DEBUG")) fprintf(stderr, "sparse24_b200: CUDA error %d: %s\n", (int)e, cudaGetErrorString(e));
    return SP24_ERR_CUDA;
}

int runtime_error() {
    launch_status();
    return SP24_ERR_CUDA;
}

}  // namespace sp24

extern "C" const char *sp24_strerror(int code) {
    switch (code) {
        case SP24_OK: return "ok";
        case SP24_ERR_SHAPE: return "unsupported shape: a dimension is not a positive multiple of the required block size";
        case SP24_ERR_STRIDE: return "unsupported leading dimension: too small or not a multiple of 16 bytes";
        case SP24_ERR_DTYPE: return "unsupported element type combination";
        case SP24_ERR_ALIGN: return "pointer is not 16-byte aligned";
        case SP24_ERR_ARG: return "invalid argument: null pointer, contradictory flags or value out of range";
        case SP24_ERR_CUDA: return "the CUDA runtime reported an error";
        case SP24_ERR_DEVICE: return "the current device is not a compute capability 10.x GPU";
        case SP24_ERR_TOO_LARGE: return "size exceeds a fixed capacity of this entry point";
        default: return "unknown sparse24_b200 error code";
    }
}

extern "C" int sp24_abi_version(void) { return SP24_ABI_VERSION; }

namespace sp24 {
namespace {
__global__ void __launch_bounds__(256) clear_kernel(uint32_t *dst, int64_t words) {
    chain_enter();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < words; i += (int64_t)gridDim.x * 256) dst[i] = 0;
}
}  // namespace

int resident_blocks(const void *kern, unsigned threads, size_t smem) {
    struct Known {
        const void *kern;
        unsigned threads;
        size_t smem;
        int blocks;
    };
    static thread_local Known known[64];      // by a hash of the kernel's address; what falls together is asked for again
    Known &k = known[(reinterpret_cast<uintptr_t>(kern) >> 4) * 0x9E3779B97F4A7C15ull >> 58];
    if (k.kern != kern || k.threads != threads || k.smem != smem) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, (int)threads, smem) != cudaSuccess) runtime_error();
        k = {kern, threads, smem, n};
    }
    return k.blocks;
}

int clear_words(void *dst, int64_t words, cudaStream_t st) {
    launch_chained(st, clear_kernel, (unsigned)((words + 1023) / 1024), 256, 0, static_cast<uint32_t *>(dst), words);
    return launch_status();
}
}  // namespace sp24

// Small buffers in the current device's memory are cleared by a kernel: a memset in the stream ends the overlap of the kernels around
// it (launch_chained).  The runtime's memset keeps what a kernel of this device may not be able to reach: memory of the host, of another
// device or managed, and pointers that the runtime does not know.
extern "C" int sp24_zero(void *dst, int64_t bytes, void *stream) {
    if (!dst || bytes < 0) return SP24_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (bytes > 0 && bytes <= 1 << 18 && bytes % 4 == 0 && (reinterpret_cast<uintptr_t>(dst) & 3u) == 0) {
        cudaPointerAttributes at{};
        int dev = -1;
        const bool known = cudaGetDevice(&dev) == cudaSuccess && cudaPointerGetAttributes(&at, dst) == cudaSuccess;
        if (!known) sp24::runtime_error();      // the memset says what is wrong
        if (known && at.type == cudaMemoryTypeDevice && at.device == dev && sp24::check_device() == SP24_OK)
            return sp24::clear_words(dst, bytes / 4, st);
    }
    if (cudaMemsetAsync(dst, 0, (size_t)bytes, st) == cudaSuccess) return SP24_OK;
    return sp24::runtime_error();
}

// Peer memory for exchanges that run on the copy engines: a buffer exported by its owner (cudaIpcGetMemHandle, or a
// framework's equivalent) is mapped into this process; copies from the returned address are ordinary device-to-device
// copies on a stream of the current device.
extern "C" int sp24_ipc_open(const void *handle, int handle_bytes, void **ptr) {
    if (!handle || !ptr || handle_bytes != (int)sizeof(cudaIpcMemHandle_t)) return SP24_ERR_ARG;
    if (int rc = sp24::check_device()) return rc;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, sizeof(h));
    *ptr = nullptr;
    if (cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess) != cudaSuccess) return sp24::runtime_error();
    return SP24_OK;
}

extern "C" int sp24_ipc_close(void *ptr) {
    if (!ptr) return SP24_ERR_ARG;
    return cudaIpcCloseMemHandle(ptr) == cudaSuccess ? SP24_OK : sp24::runtime_error();
}
