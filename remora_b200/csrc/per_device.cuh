// Answers to N yes-or-no questions about a device, each asked once per device and kept.
#pragma once
#include <atomic>

namespace rc {

// What a kernel may use (shared memory, cluster sizes) is set and asked for on the current device:
// an answer holds for that device alone. For static objects; safe with several threads, which may
// ask the same twice.
template <int N>
class PerDevice {
public:
    template <class Ask>
    bool get(int device, int question, Ask ask) {
        if (device < 0 || device >= kDevices) return ask();
        std::atomic<int>& known = known_[device][question];
        int k = known.load(std::memory_order_acquire);
        if (k == 0) {
            k = ask() ? 1 : 2;
            known.store(k, std::memory_order_release);
        }
        return k == 1;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<int> known_[kDevices][N];  // 0: not asked, 1: yes, 2: no
};

}  // namespace rc
