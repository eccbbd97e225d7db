// What has been done once for each device.  A kernel's attributes (shared memory beyond 48 KB) hold for the device that was current when
// they were set: a process that goes on to a second one must set them there too.
#pragma once
#include <atomic>

struct DeviceMarks {
    std::atomic<unsigned long long> bits{0};
    // (devices beyond the 64 are never marked: what is done once is then done every time)
    bool has(int device) const { return device >= 0 && device < 64 && (bits.load(std::memory_order_acquire) >> device & 1ull); }
    void set(int device) { if (device >= 0 && device < 64) bits.fetch_or(1ull << device, std::memory_order_release); }
    // do_it() on a device that is not marked, which it then is unless do_it() fails (returns anything but 0)
    template <typename F> int once(int device, F do_it) {
        if (has(device)) return 0;
        const int status = do_it();
        if (status == 0) set(device);
        return status;
    }
};
