/*
 * per_device.h -- what has to be done once on each device of a process, a
 * kernel's attributes for one: they belong to a device's context, so a process
 * that goes on to another GPU sets them there too.
 */
#ifndef PCA_PER_DEVICE_H
#define PCA_PER_DEVICE_H

#include <atomic>
#include <stdint.h>

namespace pcagb {

class OncePerDevice {
    std::atomic<uint64_t> done{0};   /* bit d: done on device d */

public:
    /* f() unless it has succeeded on this device before (two threads that
       come first together both call it); its success. */
    template <class F>
    bool run(int device, F &&f)
    {
        const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
        if (done.load(std::memory_order_acquire) & bit) return true;
        if (!f()) return false;
        done.fetch_or(bit, std::memory_order_release);
        return true;
    }
};

}  // namespace pcagb

#endif
