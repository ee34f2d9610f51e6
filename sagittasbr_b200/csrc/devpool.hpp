// devpool.hpp -- device memory of scenes, plans and calls.
#pragma once

#include <cstddef>

#include "common.hpp"

namespace sbr {

// A block of device memory from the device's pool; `device` is the current device.
// It may be used on any stream as soon as the call returns.
cudaError_t pool_alloc(int device, void** p, size_t bytes);
template <class T>
cudaError_t pool_alloc(int device, T** p, size_t bytes) {
    return pool_alloc(device, reinterpret_cast<void**>(p), bytes);
}
// Gives a block back (null: nothing).  All work that uses it has completed.
void pool_free(int device, void* p);
// Scenes open and close the pool of their device: what it may keep unused.
void pool_open(int device);
void pool_close(int device);

// Parts of one block: sizes first, then the addresses.
class Parts {
  public:
    size_t add(size_t bytes) {
        const size_t at = size_;
        size_ = (size_ + bytes + 255) / 256 * 256;
        return at;
    }
    size_t size() const { return size_ ? size_ : 256; }

  private:
    size_t size_ = 0;
};

}  // namespace sbr
