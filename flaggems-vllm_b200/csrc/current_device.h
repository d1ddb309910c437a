// The device guard of the native front ends (host_calls.cpp), left out where it would change nothing.  It is looked at once a call, for its
// outputs and its launch together: norms 3.56 us of the host, group quantiser 3.40, a call without outputs 2.2.  Asked for each output and the
// launch apart, both of torch and of the runtime, it costs 0.06 to 0.17 us more.
#pragma once

#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>

namespace dsv4 {

// Whether a launch of this thread goes to `device` as things are.
inline bool launches_on(c10::DeviceIndex device) {
    int at = -1;
    return cudaGetDevice(&at) == cudaSuccess && at == device;
}

// Whether an allocation does as well.  torch has to say so too: a torch guard that gives back a device without a primary context only notes
// it (per thread), and until something applies the note torch's current_device(), which its allocator goes by, is that device while the
// runtime's is another.
inline bool is_current(c10::DeviceIndex device) { return launches_on(device) && c10::cuda::current_device() == device; }

// The device of a call's tensors, current for launches and allocations, or for launches alone, as long as this lives.
class OnDevice {
   public:
    enum Use { kAllocatesToo, kLaunchesOnly };
    explicit OnDevice(c10::DeviceIndex device, Use use = kAllocatesToo) : index(device) {
        if (!(use == kAllocatesToo ? is_current(device) : launches_on(device))) guard_.set_device(c10::Device(c10::kCUDA, device));
    }
    const c10::DeviceIndex index;

   private:
    c10::cuda::OptionalCUDAGuard guard_;
};

// f() with `device` current.
template <typename F>
auto with_device(c10::DeviceIndex device, F&& f) {
    const OnDevice here(device);
    return f();
}

}  // namespace dsv4
