// Values per device, made at their first use and kept for the life of the process.
#pragma once
#include <atomic>
#include <memory>
#include <mutex>
#include <utility>

namespace ssb {

// get() may be called by several threads at once: the threads that run a backward hold no interpreter lock.  Every caller gets
// the same value, complete.  `make` runs outside the lock, so a thread that makes a value waits for no other one (an allocation
// may want the interpreter lock, which another maker may hold); of several values made at the same time one is kept.
template <class T, int kDevices = 64>
class PerDevice {
 public:
  template <class Make>
  T& get(int device, Make make) {
    Slot& s = slots_[device];
    if (T* ready = s.ready.load(std::memory_order_acquire)) return *ready;
    auto made = std::make_unique<T>(make());
    std::lock_guard<std::mutex> hold(s.lock);
    if (!s.value) {
      s.value = std::move(made);
      s.ready.store(s.value.get(), std::memory_order_release);
    }
    return *s.value;
  }

 private:
  struct Slot {
    std::atomic<T*> ready{nullptr};
    std::mutex lock;
    std::unique_ptr<T> value;
  };
  Slot slots_[kDevices];
};

// A positive number per device that the CUDA runtime is asked for once, or what has to be set there once (a kernel's attributes
// belong to a device).  `make(int* value)` returns an error code, which is handed on and not kept; threads that come together
// may each ask.  A value of 0 means: not asked yet.
template <int kDevices = 64>
class OncePerDevice {
 public:
  template <class Make>
  int get(int device, int* value, Make make) {
    std::atomic<int>& kept = values_[device];
    if ((*value = kept.load(std::memory_order_acquire)) != 0) return 0;
    const int rc = make(value);
    if (rc == 0) kept.store(*value, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<int> values_[kDevices] = {};
};

}  // namespace ssb
