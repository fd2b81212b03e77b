// Work that has to be done once per device of a process, such as raising a
// kernel's shared-memory limit: several host threads may each drive a device.

#ifndef SLQ_ONCE_H_
#define SLQ_ONCE_H_

#include <atomic>
#include <cstdint>

namespace slq {

class DeviceOnce {
public:
    // setup() unless it has succeeded for this device (0 is success).  Two
    // threads that come first together both run it.
    template <typename F>
    int operator()(int device, F setup)
    {
        if (device < 0 || device >= 64) return setup();
        const uint64_t bit = uint64_t(1) << device;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int status = setup();
        if (status == 0) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace slq

#endif  // SLQ_ONCE_H_
