// Host state that belongs to a device.  A kernel's attributes (its limit of shared memory, cluster sizes beyond 8) and what the driver
// says about its residency hold for the device that was current when they were set or asked; a process may use several.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

// A number for each device, 0 until it is set: of the current device, from any thread.  Devices beyond the table keep none (callers do
// their work again).
class PerDevice {
public:
    int get() {
        std::atomic<int>* value = of_current();
        return value ? value->load(std::memory_order_acquire) : 0;
    }
    void set(int x) {
        if (std::atomic<int>* value = of_current()) value->store(x, std::memory_order_release);
    }

private:
    static constexpr int DEVICES = 64;
    std::atomic<int> values[DEVICES] = {};
    std::atomic<int>* of_current() {
        int device = 0;
        return cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < DEVICES ? &values[device] : nullptr;
    }
};
