// Small pinned host buffers shared by a process's handles.
//
// A read-back into pinned memory saves 4.5 us (62.1 -> 57.6 us for a reduction
// and a resampling of 1000 particles), but pinning takes 2.4 ms and releasing
// it 0.4 ms (B200 host), which a handle that is used a few times never earns
// back: a resampler made, used once and dropped took 3.3 ms with a buffer of
// its own against 0.8 ms.  So the process pins one block at the first use and
// keeps it to its end; handles borrow its slots and return them.  The block
// does not grow: a handle that finds every slot taken does without.
#pragma once
#include <cstddef>
#include <mutex>

namespace bpf {

// T: what a slot holds; N: slots of the block.  alloc pins `bytes` (null when
// it cannot), valid says whether a block still is what alloc returned (a reset
// of the device takes it away).  Safe from any number of threads.
template <class T, int N>
class HostSlots {
 public:
  using Alloc = void* (*)(size_t bytes);
  using Valid = bool (*)(void* block);
  HostSlots(Alloc alloc, Valid valid) : alloc_(alloc), valid_(valid) {}

  // a slot of the caller's own, or null
  T* acquire() {
    std::lock_guard<std::mutex> lk(mu_);
    if (block_ && !valid_(block_)) {  // the slots in use went with it
      block_ = nullptr;
      for (bool& t : taken_) t = false;
    }
    if (!block_) block_ = static_cast<T*>(alloc_(N * sizeof(T)));
    if (!block_) return nullptr;
    for (int i = 0; i < N; ++i)
      if (!taken_[i]) {
        taken_[i] = true;
        return block_ + i;
      }
    return nullptr;
  }

  // nothing may still write to the slot
  void release(T* slot) {
    if (!slot) return;
    std::lock_guard<std::mutex> lk(mu_);
    for (int i = 0; block_ && i < N; ++i)
      if (slot == block_ + i) taken_[i] = false;
  }

 private:
  Alloc alloc_;
  Valid valid_;
  std::mutex mu_;
  T* block_ = nullptr;
  bool taken_[N] = {};
};

}  // namespace bpf
