// scratch.hpp — working arrays of one build, carved from a few pieces of memory.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace eikgb {

// Alloc: bool get(void** p, size_t bytes) and void put(void* p).
//
// A build asks for some 45 arrays; allocating and releasing them one by one took 1.2 of
// the 2.5 ms that a 33^3 cube's takes.  Arrays below kLarge share pieces, each as large as
// all before it, from kFirst up to kMost bytes.  Larger arrays have a piece of exactly
// their size: there the allocation is a small part of the work, and the build of a mesh
// that nearly fills the GPU must not ask for more than it uses.  Where a shared piece
// cannot be had, the array alone is asked for.
template <class Alloc>
class ScratchPieces {
 public:
  static constexpr size_t kFirst = (size_t)8 << 20, kMost = (size_t)32 << 20, kLarge = (size_t)16 << 20;
  explicit ScratchPieces(Alloc a = Alloc()) : alloc_(a) {}
  ~ScratchPieces() {
    for (void* p : pieces_) alloc_.put(p);
  }
  ScratchPieces(const ScratchPieces&) = delete;
  ScratchPieces& operator=(const ScratchPieces&) = delete;

  // `size` bytes at a 256-byte boundary, or null
  void* get(size_t size) {
    const size_t bytes = (std::max<size_t>(size, 1) + 255) & ~(size_t)255;
    if (bytes <= left_) {
      void* p = at_;
      at_ += bytes;
      left_ -= bytes;
      return p;
    }
    if (bytes < kLarge) {
      const size_t piece = std::max(bytes, std::min(kMost, std::max(kFirst, total_)));
      if (void* q = own(piece)) {
        at_ = static_cast<unsigned char*>(q) + bytes;
        left_ = piece - bytes;
        return q;
      }
    }
    return own(bytes);
  }

 private:
  void* own(size_t bytes) {
    void* q = nullptr;
    pieces_.reserve(pieces_.size() + 1);
    if (!alloc_.get(&q, bytes)) return nullptr;
    pieces_.push_back(q);
    total_ += bytes;
    return q;
  }
  Alloc alloc_;
  std::vector<void*> pieces_;
  unsigned char* at_ = nullptr;  // unused rest of the last shared piece
  size_t left_ = 0, total_ = 0;
};

}  // namespace eikgb
