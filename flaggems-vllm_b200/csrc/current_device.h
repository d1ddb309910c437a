// The device guard of the native front ends (host_calls.cpp), left out where it would change nothing: a call with two outputs then takes
// 3.55 us of the host instead of 3.9.  Asking the runtime as well as torch costs less than runs differ (norms 3.96-4.01 and 3.99-4.00 us).
#pragma once

#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>

namespace dsv4 {

// Whether a launch or an allocation of this thread goes to `device` as things are.  Both torch and the CUDA runtime have to say so: a torch
// guard that gives back a device without a primary context only notes it (per thread), and until something applies the note torch's
// current_device() is that device while the runtime's is another.
inline bool is_current(c10::DeviceIndex device) {
    int at = -1;
    return c10::cuda::current_device() == device && cudaGetDevice(&at) == cudaSuccess && at == device;
}

// f() with `device` current.
template <typename F>
auto with_device(c10::DeviceIndex device, F&& f) {
    c10::cuda::OptionalCUDAGuard guard;
    if (!is_current(device)) guard.set_device(c10::Device(c10::kCUDA, device));
    return f();
}

}  // namespace dsv4
