// A buffer that a caller can do without (the records of handed-over cells): a request that was
// refused is not made again at that size or above, and a smaller buffer stays until a larger one is there.
#ifndef PGB_OPTIONAL_BUFFER_H
#define PGB_OPTIONAL_BUFFER_H

#include <cstddef>

namespace pgb_host {

struct OptionalBuffer {
  void* p = nullptr;
  size_t cap = 0, refused = 0;  // refused: smallest request that failed (0: none)

  // True if `bytes` fit. alloc(bytes) returns null on failure; replaced(old) is called before p changes,
  // and disposes of `old` (null the first time).
  template <class Alloc, class Replaced>
  bool ensure(size_t bytes, Alloc alloc, Replaced replaced) {
    if (bytes <= cap) return true;
    if (refused && bytes >= refused) return false;
    void* q = alloc(bytes);
    if (!q) {
      refused = bytes;
      return false;
    }
    replaced(p);
    p = q;
    cap = bytes;
    return true;
  }
};

}  // namespace pgb_host

#endif  // PGB_OPTIONAL_BUFFER_H
