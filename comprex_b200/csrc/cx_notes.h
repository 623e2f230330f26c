// What the kernel launched last on a stream of this library is like, for the kernel about to be launched
// behind it: does it let that one in before it has finished (cx_device.cuh)?  Plain C++, no CUDA.
#pragma once
#include <stdint.h>

#include <atomic>
#include <mutex>

class CxStreamNotes {
 public:
  static constexpr int kDevices = 64, kSlots = 64;

  void note(int dev, const void* stream, bool early) {
    if (known(dev, stream)) slot(dev, stream).store(word(stream, early), std::memory_order_relaxed);
  }
  // Held from the question or the note to the launch it is about: the notes of a stream are in the order of
  // its kernels then, also where several threads share the stream.
  std::mutex& order(int dev, const void* stream) {
    return known(dev, stream) ? order_[dev][index(stream)] : order_of_others_;
  }
  // true unless the last note of this very stream says "not early"
  bool front_wait(int dev, const void* stream) const {
    return !known(dev, stream) || slot(dev, stream).load(std::memory_order_relaxed) != word(stream, false);
  }

 private:
  // A handle names a stream only together with its device (the default stream is 0 on all of them); the
  // per-thread default stream, 2, is another stream in every thread; 1 is the default stream once more.
  static bool known(int dev, const void* stream) {
    return dev >= 0 && dev < kDevices && reinterpret_cast<uint64_t>(stream) != 2;
  }
  static uint64_t handle(const void* stream) {
    const uint64_t s = reinterpret_cast<uint64_t>(stream);
    return s == 1 ? 0 : s;
  }
  static uint64_t word(const void* stream, bool early) { return handle(stream) << 2 | 2u | (early ? 1u : 0u); }
  // hashed: what another stream has overwritten counts as early
  std::atomic<uint64_t>& slot(int dev, const void* stream) const {
    return last_[dev][index(stream)];
  }
  static unsigned index(const void* stream) {
    const uint64_t s = handle(stream);
    return (unsigned)((s >> 4 ^ s >> 10 ^ s >> 16) % kSlots);
  }
  mutable std::atomic<uint64_t> last_[kDevices][kSlots] = {};
  std::mutex order_[kDevices][kSlots], order_of_others_;
};
