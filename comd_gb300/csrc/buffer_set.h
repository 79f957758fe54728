// buffer_set.h -- buffers that are replaced together or not at all.
#pragma once

#include <cstddef>

namespace cg {

// N buffers with the bytes each was allocated with.  reserve makes every buffer
// at least bytes[q] large (contents are not kept where one is replaced).  When an
// allocation fails the ones made so far are given back and the set is as it was.
// alloc(bytes) returns null on failure; the caller owns the buffers (release).
template <int N>
struct BufferSet {
  void *buf[N] = {};
  size_t cap[N] = {};

  template <class Alloc, class Free>
  bool reserve(const size_t (&bytes)[N], Alloc &&alloc, Free &&free) {
    void *fresh[N] = {};
    for (int q = 0; q < N; q++) {
      if (buf[q] && bytes[q] <= cap[q]) continue;
      fresh[q] = alloc(bytes[q] > 0 ? bytes[q] : 1);
      if (fresh[q]) continue;
      for (int k = 0; k < q; k++)
        if (fresh[k]) free(fresh[k]);
      return false;
    }
    for (int q = 0; q < N; q++)
      if (fresh[q]) {
        if (buf[q]) free(buf[q]);
        buf[q] = fresh[q];
        cap[q] = bytes[q];
      }
    return true;
  }
  template <class Free>
  void release(Free &&free) {
    for (int q = 0; q < N; q++) {
      if (buf[q]) free(buf[q]);
      buf[q] = nullptr;
      cap[q] = 0;
    }
  }
};

}  // namespace cg
