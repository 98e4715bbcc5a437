// What a launcher sets up once for its kernel: the opt-in to more shared memory than 48 KB
// and the number of CTAs the chip holds at once.  Both belong to a device, so they
// are kept per device; host threads may launch at the same time.
#pragma once
#include <atomic>

namespace fcb {

// N numbers per device, made by setup(int* out) -> error (0: success) at the first call for
// a device.  Two threads that come first at once both run setup, which gives both the same
// numbers; a setup that failed runs again at the next call.
template <int N = 1>
class PerDevice {
  public:
    static constexpr int kDevices = 64;  // devices beyond these run setup on every call
    template <class F>
    auto get(int device, int* out, const F& setup) -> decltype(setup(out)) {
        const bool kept = device >= 0 && device < kDevices;
        if (kept && done_[device].load(std::memory_order_acquire)) {
            for (int k = 0; k < N; ++k) out[k] = value_[device][k].load(std::memory_order_relaxed);
            return decltype(setup(out))(0);
        }
        const auto e = setup(out);
        if (e == decltype(setup(out))(0) && kept) {
            for (int k = 0; k < N; ++k) value_[device][k].store(out[k], std::memory_order_relaxed);
            done_[device].store(true, std::memory_order_release);
        }
        return e;
    }

  private:
    std::atomic<int> value_[kDevices][N]{};
    std::atomic<bool> done_[kDevices]{};
};

}  // namespace fcb

#ifdef __CUDACC__
#include <cuda_runtime.h>

namespace fcb {

// CTAs of `kernel` that the current device holds at once, launched with `bytes` of
// dynamic shared memory (opted in to); at least 1.
template <class K>
cudaError_t resident_ctas(K kernel, int threads, size_t bytes, int* out) {
    int dev = 0, sms = 0, occ = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, bytes);
    if (e == cudaSuccess) *out = sms * occ > 0 ? sms * occ : 1;
    return e;
}

// PerDevice::get for the current device.
template <int N, class F>
cudaError_t per_device(PerDevice<N>& kept, int* out, const F& setup) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e != cudaSuccess ? e : kept.get(dev, out, setup);
}

}  // namespace fcb
#endif
