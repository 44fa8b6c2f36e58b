// A value that is found out once for each device and kept: an attribute set, a launch shape.  Any
// thread may ask; threads that ask at the same time may each find it out, to the same value.
#pragma once
#include <atomic>
#include <cstddef>
#include <initializer_list>

#include <cuda_runtime_api.h>

namespace cc {

class PerDevice {
    static constexpr int MAX_DEVICES = 64;
    std::atomic<int> value_[MAX_DEVICES] = {};

public:
    // find(): the value for the current device; kept when it is above 0, asked for again otherwise
    template <class F>
    int get(F &&find) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return find();
        int v = value_[dev].load(std::memory_order_acquire);
        if (v > 0) return v;
        v = find();
        if (v > 0) value_[dev].store(v, std::memory_order_release);
        return v;
    }
};

// the kernels may use this much dynamic shared memory; for PerDevice::get
template <class... K>
int allow_shared(size_t bytes, K... kernels) {
    bool ok = true;
    for (cudaError_t e : {cudaFuncSetAttribute((const void *)kernels, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)bytes)...})
        ok = ok && e == cudaSuccess;
    return ok ? 1 : 0;
}

}  // namespace cc
