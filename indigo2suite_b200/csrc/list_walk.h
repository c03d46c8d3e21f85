// Walks over the entries of a CSR list (host and device).
//
// A graph may hold INT_MAX entries, so a list may end at INT_MAX, and a cursor
// that steps by a warp, a block or a window of entries past such an end does
// not fit an int: it would turn negative, stay below the end and read before
// the array. Positions are unsigned here; with ends of at most 2^31 - 1 and
// steps far below 2^31 they never wrap.
#pragma once
#include "host_device.h"

namespace i2 {

// f(j) for the positions begin + first, + step, + 2 step, ... below end.
template <class F>
I2_HOST_DEVICE void walk_list(unsigned begin, unsigned end, unsigned first, unsigned step, F f) {
  for (unsigned j = begin + first; j < end; j += step) f(j);
}

// A group of `width` threads reads a list in windows of 4 * width entries,
// thread t the entries k + t, k + t + width, ... of the window at k < end:
// how many of its four lie below end.
I2_HOST_DEVICE int window_share(unsigned k, unsigned end, unsigned t, unsigned width) {
  const unsigned left = end - k;
  if (left <= t) return 0;
  const unsigned n = (left - t + width - 1) / width;
  return (int)(n < 4u ? n : 4u);
}

}  // namespace i2
