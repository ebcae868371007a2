// Clearing a film, shared with a host-side test that stands in for the CUDA runtime.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace gr {

// Makes `device` the calling thread's device for a scope.
struct DeviceScope {
    int before = -1;
    cudaError_t status;
    explicit DeviceScope(int device) {
        int now = device;
        status = cudaGetDevice(&now);
        if (status != cudaSuccess || now == device) return;
        status = cudaSetDevice(device);
        if (status == cudaSuccess) before = now;
    }
    DeviceScope(const DeviceScope&) = delete;
    DeviceScope& operator=(const DeviceScope&) = delete;
    ~DeviceScope() {
        if (before >= 0) cudaSetDevice(before);
    }
};

// Zeroes a film's pixels, and its splats if it has them, on the default stream of its device
// and records `cleared` there, which renders on other streams wait for.  CUDA takes an event
// and a stream of one device only, and the caller may have another one current.
inline cudaError_t clear_film(int device, void* pixels, void* splat, size_t bytes, cudaEvent_t cleared) {
    const DeviceScope on(device);
    cudaError_t e = on.status;
    if (e == cudaSuccess) e = cudaMemset(pixels, 0, bytes);
    if (e == cudaSuccess && splat) e = cudaMemset(splat, 0, bytes);
    if (e == cudaSuccess) e = cudaEventRecord(cleared, 0);
    return e;
}

}  // namespace gr
