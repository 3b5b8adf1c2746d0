// smem_limit.h — how much dynamic shared memory each kernel has been allowed,
// by device.
//
// The limit (cudaFuncAttributeMaxDynamicSharedMemorySize) belongs to the kernel
// and the device, the size to the launch.  Were it set to each launch's size, a
// smaller launch (another context's K, another thread) would take away what a
// larger one needs between its own setting and its launch, or when a context
// captures its graphs again.  So it is only ever raised.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <new>
#include <utility>

namespace culda {

class SmemLimits {
  public:
    // Raises the limit of `fn` on `device` to `bytes` unless it is that high;
    // set(bytes) sets it and returns 0 or its status.
    template <class Set>
    int raise(const void *fn, int device, size_t bytes, int no_memory, Set set) {
        std::lock_guard<std::mutex> lock(mu_);
        try {
            size_t &have = have_[{fn, device}];
            if (have >= bytes) return 0;
            const int status = set(bytes);
            if (status == 0) have = bytes;
            return status;
        } catch (const std::bad_alloc &) {
            return no_memory;
        }
    }

  private:
    std::mutex mu_;
    std::map<std::pair<const void *, int>, size_t> have_;
};

}  // namespace culda
