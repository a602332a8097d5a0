// Stream-ordered scratch memory for kernels that split one call over several launches.
//
// The buffers come from a memory pool of this library, one per device, through the stream-ordered
// allocator: a buffer is usable by the work queued after it on its stream and goes back to the pool
// behind that work, so calls on several streams and threads never share one by accident.  The pool keeps
// at most kScratchKept bytes between calls (what lies above goes back to the device at the next
// synchronisation), and everything when the process ends.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace mega {

constexpr size_t kScratchKept = size_t(256) << 20;

void* scratch_alloc(size_t bytes, cudaStream_t s);  // nullptr when the device refuses
void scratch_free(void* p, cudaStream_t s);

// One call's scratch: carved into 256-byte aligned pieces, given back (behind the queued work) on scope exit.
class Scratch {
 public:
  Scratch(size_t bytes, cudaStream_t s) : s_(s), base_(static_cast<char*>(scratch_alloc(bytes, s))), left_(bytes) {
    cur_ = base_;
  }
  ~Scratch() {
    if (base_) scratch_free(base_, s_);
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  explicit operator bool() const { return base_ != nullptr; }
  static constexpr size_t padded(size_t bytes) { return (bytes + 255) & ~size_t(255); }
  template <typename T>
  T* take(size_t n) {
    const size_t b = padded(n * sizeof(T));
    if (!base_ || b > left_) return nullptr;
    T* p = reinterpret_cast<T*>(cur_);
    cur_ += b;
    left_ -= b;
    return p;
  }

 private:
  cudaStream_t s_;
  char* base_;
  char* cur_ = nullptr;
  size_t left_;
};

}  // namespace mega
