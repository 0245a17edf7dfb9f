// Shared host helpers of the C ABI: error reporting, device buffers, handles.
#pragma once

#include "emp_b200.h"
#include "emp_compact.h"
#include "emp_model.h"

#include <cuda_runtime.h>

#include <string>
#include <utility>

namespace emp {

std::string& last_error();
void clear_error();
emp_status fail(emp_status status, const std::string& message);
emp_status cuda_fail(cudaError_t e, const char* what);
// Makes `device` current (-1: keep the current one) and reports its ordinal.
emp_status select_device(int device, int* ordinal);

// Device memory comes from a pool of this library's own, one per device, that holds on to at most
// kPoolKeep bytes of freed memory between calls (the driver takes unused pool memory back when an
// allocation elsewhere in the process would fail).  Blocks above kPoolBlock are not pooled:
// mapping and unmapping them under the pool's limit took up to a second.  cudaMalloc and cudaFree cost
// 0.1 to 0.3 ms a pair on a B200 and a one-shot count makes some thirty: a 5x5 count took 6.5 ms,
// 0.04 ms of it on the device.  Like cudaFree, device_free waits for the device, so no stream still uses what
// goes back.  Safe from several threads; a device reset in between is noticed.  device_trim gives all
// that is unused in the current device's pool back to the driver.
constexpr uint64_t kPoolKeep = 2ull << 30, kPoolBlock = 512ull << 20;
cudaError_t device_alloc(void** p, size_t bytes, int* device, uint64_t* context);
void device_free(void* p, int device, uint64_t context);
cudaError_t device_trim();

// Owning device allocation (move-only).
struct DeviceBuffer {
    void* p = nullptr;
    size_t bytes = 0;
    int device = 0;
    uint64_t context = 0;
    DeviceBuffer() = default;
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    DeviceBuffer(DeviceBuffer&& o) noexcept { take(o); }
    DeviceBuffer& operator=(DeviceBuffer&& o) noexcept
    {
        if (this != &o) {
            release();
            take(o);
        }
        return *this;
    }
    ~DeviceBuffer() { release(); }
    void release()
    {
        if (p) device_free(p, device, context);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t alloc(size_t n)
    {
        release();
        bytes = n;
        return n ? device_alloc(&p, n, &device, &context) : cudaSuccess;
    }
    // Keeps the allocation when it holds n bytes already (a free waits for the whole device,
    // which would stall work queued on other streams).
    cudaError_t reserve(size_t n) { return n <= bytes && p ? cudaSuccess : alloc(n); }
    template <class T>
    T* as() const { return static_cast<T*>(p); }

private:
    void take(DeviceBuffer& o)
    {
        p = o.p;
        bytes = o.bytes;
        device = o.device;
        context = o.context;
        o.p = nullptr;
        o.bytes = 0;
    }
};

}  // namespace emp

struct emp_puzzle_t {
    emp::PuzzleModel model;
    std::vector<uint32_t> order;
    std::vector<emp::LevelPlan> plan;
    emp::DeviceTables tables;
    std::vector<uint32_t> compact;  // compact search tables; empty when the puzzle has none
    uint32_t extra_count = 0;
};

#define CUDA_TRY(expr)                                       \
    do {                                                     \
        cudaError_t e_ = (expr);                             \
        if (e_ != cudaSuccess) return emp::cuda_fail(e_, #expr); \
    } while (0)

#define EMP_TRY(expr)                       \
    do {                                    \
        emp_status s_ = (expr);             \
        if (s_ != EMP_OK) return s_;        \
    } while (0)
