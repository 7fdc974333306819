// pms_per_device.h -- values that belong to a device (kernel attributes set there, what it holds at once),
// made on the first use of each device and kept until the process exits.
#pragma once
#include <mutex>

namespace pms {

// At most MAXDEV devices, one T each; safe with several host threads (the first use of a device makes its
// value while the others wait).
template <class T, int MAXDEV = 64>
class PerDevice {
  public:
    // The value of device `dev`, made by make(T&) unless it is there.  make returns whether it succeeded; a value
    // that failed is not kept (the next call tries again).  False: not made, or no such device number.
    template <class F>
    bool get(int dev, T& out, F&& make) {
        if (dev < 0 || dev >= MAXDEV) return false;
        std::lock_guard<std::mutex> lock(m_);
        if (!have_[dev]) {
            T v{};
            if (!make(v)) return false;
            value_[dev] = v;
            have_[dev] = true;
        }
        out = value_[dev];
        return true;
    }

  private:
    std::mutex m_;
    T value_[MAXDEV] = {};
    bool have_[MAXDEV] = {};
};

}  // namespace pms
