// What is set up once per GPU of the process, by the first call on it: kernel
// attributes and what follows from them belong to a device.  Safe with
// several threads (two first calls at once both do the work).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace sddc {

class PerDevice {
  public:
    // the device's value (positive): made by make(device, &value) where it is not there yet
    template <typename F> cudaError_t get(int *out, F make)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const bool kept = dev >= 0 && dev < kDevices;  // (beyond: made every time)
        if (kept && (*out = value_[dev].load(std::memory_order_acquire)) > 0) return cudaSuccess;
        e = make(dev, out);
        if (e == cudaSuccess && kept) value_[dev].store(*out, std::memory_order_release);
        return e;
    }

  private:
    static constexpr int kDevices = 64;
    std::atomic<int> value_[kDevices] = {};
};

// the dynamic shared memory of kernels, and the whole unified L1/shared array as
// shared memory, so that several CTAs fit on an SM
template <typename K> cudaError_t set_smem(K kern, size_t bytes)
{
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}

// CTAs of a kernel resident at once on a device; sets its attributes on the way
template <typename K> cudaError_t resident_ctas(K kern, int threads, size_t smem, int dev, int *n)
{
    int sms = 0, per_sm = 0;
    cudaError_t e = set_smem(kern, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    *n = sms * per_sm > 1 ? sms * per_sm : 1;
    return e;
}

}  // namespace sddc
