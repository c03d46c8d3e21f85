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

// f(j) for the positions begin + first, + step, + 2 step, ... below end. Counted,
// not compared with the end: a loop over unsigned positions may wrap as far as the
// compiler knows, and it would then not issue the loads of several steps together
// (union-find on a star whose hub comes last, us: 64 by comparison, 54 counted).
template <class F>
I2_HOST_DEVICE void walk_list(unsigned begin, unsigned end, unsigned first, unsigned step, F f) {
  const unsigned from = begin + first;
  const unsigned n = from < end ? (end - from + step - 1) / step : 0;
  for (unsigned i = 0; i < n; ++i) f(from + i * step);
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
