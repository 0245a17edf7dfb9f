// Shared host helpers of the C ABI (emp_common.h).
#include "emp_common.h"

#include <cuda.h>

#include <map>
#include <mutex>

namespace emp {

namespace {

// Identity of the current context: a device reset makes a new one, with other memory.
uint64_t context_id()
{
    using Fn = CUresult (*)(CUcontext, unsigned long long*);
    static const Fn get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess) f = nullptr;
        return reinterpret_cast<Fn>(f);
    }();
    unsigned long long id = 0;
    if (!get) return 0;
    if (get(nullptr, &id) == CUDA_SUCCESS) return id;
    cudaFree(nullptr);  // makes the device's primary context current
    return get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

struct Pool {
    cudaMemPool_t pool;
    cudaStream_t stream;  // allocations and frees are ordered on it; nothing else runs there
};

std::mutex g_pool_lock;
// by context; never destroyed: at process end the driver may be gone before this is
std::map<uint64_t, Pool>& pools()
{
    static auto* m = new std::map<uint64_t, Pool>();
    return *m;
}

// the pool of the current context; null when the device has none
Pool* current_pool(int device, uint64_t context)
{
    auto it = pools().find(context);
    if (it != pools().end()) return it->second.pool ? &it->second : nullptr;
    Pool p{};
    int supported = 0;
    cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, device);
    if (context && supported) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        uint64_t keep = kPoolKeep;
        if (cudaMemPoolCreate(&p.pool, &props) != cudaSuccess) p.pool = nullptr;
        else if (cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                 cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess) {
            cudaMemPoolDestroy(p.pool);
            p.pool = nullptr;
        }
        cudaGetLastError();
    }
    Pool& kept = pools()[context] = p;
    return kept.pool ? &kept : nullptr;
}

}  // namespace

cudaError_t device_alloc(void** out, size_t bytes, int* device, uint64_t* context)
{
    *out = nullptr;
    cudaError_t e = cudaGetDevice(device);
    if (e != cudaSuccess) return e;
    *context = 0;
    if (bytes <= kPoolBlock) {
        const uint64_t id = context_id();
        std::lock_guard<std::mutex> g(g_pool_lock);
        if (Pool* p = current_pool(*device, id)) {
            e = cudaMallocFromPoolAsync(out, bytes, p->pool, p->stream);
            if (e == cudaErrorMemoryAllocation) {  // what the pool still holds may be in the way
                cudaGetLastError();
                cudaMemPoolTrimTo(p->pool, 0);
                e = cudaMallocFromPoolAsync(out, bytes, p->pool, p->stream);
            }
            // usable from any stream from here on: nothing but the pool's own work is on its stream
            if (e == cudaSuccess && cudaStreamQuery(p->stream) != cudaSuccess) {
                cudaGetLastError();
                e = cudaStreamSynchronize(p->stream);
            }
            if (e == cudaSuccess) *context = id;
            return e;
        }
    }
    return cudaMalloc(out, bytes);
}

void device_free(void* p, int device, uint64_t context)
{
    if (!context) {
        cudaFree(p);
        return;
    }
    int now = device;
    cudaGetDevice(&now);
    if (now != device) cudaSetDevice(device);
    if (context_id() == context) {  // else a device reset took the memory along
        cudaDeviceSynchronize();
        std::lock_guard<std::mutex> g(g_pool_lock);
        cudaFreeAsync(p, pools()[context].stream);
    }
    if (now != device) cudaSetDevice(now);
}

cudaError_t device_trim()
{
    const uint64_t id = context_id();
    std::lock_guard<std::mutex> g(g_pool_lock);
    auto it = pools().find(id);
    if (it == pools().end() || !it->second.pool) return cudaSuccess;  // nothing was pooled here
    const cudaError_t e = cudaStreamSynchronize(it->second.stream);
    return e != cudaSuccess ? e : cudaMemPoolTrimTo(it->second.pool, 0);
}

std::string& last_error()
{
    thread_local std::string message;
    return message;
}

void clear_error() { last_error().clear(); }

emp_status fail(emp_status status, const std::string& message)
{
    last_error() = message;
    return status;
}

emp_status cuda_fail(cudaError_t e, const char* what)
{
    const emp_status s = e == cudaErrorMemoryAllocation ? EMP_ERR_NOMEM : EMP_ERR_CUDA;
    cudaGetLastError();  // clear a sticky-free error so the next call starts clean
    return fail(s, std::string(what) + ": " + cudaGetErrorString(e));
}

emp_status select_device(int device, int* ordinal)
{
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0)
        return fail(EMP_ERR_CUDA, std::string("no CUDA device available: ") + cudaGetErrorString(e));
    if (device >= 0) {
        if (device >= count) return fail(EMP_ERR_INVALID, "device ordinal out of range");
        e = cudaSetDevice(device);
        if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
        *ordinal = device;
    } else {
        e = cudaGetDevice(ordinal);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    }
    return EMP_OK;
}

}  // namespace emp
