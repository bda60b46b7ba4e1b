#include "common.cuh"

#include <cstdlib>
#include <mutex>

namespace macko {

char *last_error_buffer()
{
    static thread_local char buf[512] = "";
    return buf;
}

int fail(int status, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(last_error_buffer(), 512, fmt, ap);
    va_end(ap);
    return status;
}

int current_device_info(const DeviceInfo **out)
{
    static DeviceInfo infos[kMaxDevices];
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(MACKO_ERR_CUDA, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    DeviceInfo &d = infos[dev];
    if (!d.valid) {
        e = cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "cudaDeviceGetAttribute: %s", cudaGetErrorString(e));
        d.valid = true;
    }
    *out = &d;
    return MACKO_OK;
}

int check_product_args(const void *values, const void *deltas, const int32_t *ri, int64_t rows, int64_t cols,
                       int64_t padded_count, const void *x, const void *y)
{
    if (rows < 0 || cols < 0 || padded_count < 0)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "negative size (rows=%lld cols=%lld P=%lld)",
                    (long long)rows, (long long)cols, (long long)padded_count);
    if (rows >= (1LL << 31) - 64 || cols >= (1LL << 30) || padded_count >= (1LL << 31))
        return fail(MACKO_ERR_SIZE_OVERFLOW, "rows=%lld cols=%lld P=%lld exceed 31-bit indexing",
                    (long long)rows, (long long)cols, (long long)padded_count);
    if (padded_count % 8 != 0)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "padded_count %lld is not a multiple of 8", (long long)padded_count);
    if (rows == 0) return MACKO_OK;
    if (!ri || !y) return fail(MACKO_ERR_INVALID_ARGUMENT, "null row_indices or y");
    if (cols > 0 && !x) return fail(MACKO_ERR_INVALID_ARGUMENT, "null x");
    if (padded_count > 0 && (!values || !deltas)) return fail(MACKO_ERR_INVALID_ARGUMENT, "null values or deltas");
    if (!aligned(values, 16)) return fail(MACKO_ERR_MISALIGNED, "values must be 16-byte aligned");
    if (!aligned(deltas, 4)) return fail(MACKO_ERR_MISALIGNED, "deltas must be 4-byte aligned");
    if (!aligned(ri, 4)) return fail(MACKO_ERR_MISALIGNED, "row_indices must be 4-byte aligned");
    if (!aligned(x, 2) || !aligned(y, 2)) return fail(MACKO_ERR_MISALIGNED, "x and y must be 2-byte aligned");
    return MACKO_OK;
}

bool use_pdl()
{
    static const bool on = [] {
        const char *v = getenv("MACKO_SPMV_PDL");
        return !(v && v[0] == '0');
    }();
    return on;
}

}  // namespace macko

extern "C" {

int macko_version(void) { return MACKO_B200_VERSION; }

const char *macko_status_string(int status)
{
    switch (status) {
        case MACKO_OK: return "ok";
        case MACKO_ERR_INVALID_ARGUMENT: return "invalid argument";
        case MACKO_ERR_MISALIGNED: return "misaligned buffer";
        case MACKO_ERR_SIZE_OVERFLOW: return "size overflow";
        case MACKO_ERR_CUDA: return "CUDA error";
        case MACKO_ERR_WORKSPACE: return "workspace too small";
        default: return "unknown status";
    }
}

const char *macko_last_error(void) { return macko::last_error_buffer(); }
}
