// What the kernel launched last on a stream of this library is like, for the kernel about to be launched
// behind it: does it let that one in before it has finished (cx_device.cuh)?  Plain C++, no CUDA.
#pragma once
#include <stdint.h>

#include <atomic>
#include <mutex>

/* how a receive kernel waits for the kernel in front */
#define CX_WAIT_NONE 0u     /* the sender is in front, of the same native call: it touches none of the vectors */
#define CX_WAIT_START 1u    /* a kernel that was let in early may be in front: wait first */
#define CX_WAIT_VECTORS 2u  /* wait before the vectors are touched */
#define CX_WAIT_CHAIN 3u    /* like CX_WAIT_START, and the kernel behind (chained) is let in after that */

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

// What a thread's native call has launched so far, for the op it launches next.  Between two calls the program
// may queue kernels of its own on the stream, which the notes do not know: only a sender that the op in front,
// in the same call, has launched on the same stream is known to be the kernel in front.
class CxCallFront {
 public:
  void begin_call() { sent_ = behind_ = false; }
  void begin_op(const void* stream) {
    behind_ = sent_ && stream_ == stream;
    sent_ = false;
  }
  void sender(const void* stream) {
    sent_ = true;
    stream_ = stream;
  }
  void end_call() { sent_ = behind_ = false; }
  bool behind_sender() const { return behind_; }

 private:
  const void* stream_ = nullptr;
  bool sent_ = false, behind_ = false;
};
