// Sort keys of the vertex pairs of a graph (gen_device.cu).
#pragma once
#include "host_device.h"

namespace i2 {

// Keys of the vertex pairs of a graph of n vertices: `shift` bits hold an ID
// (those of n, which marks dropped pairs), and keys sort over `bits` bits.
struct KeyBits {
  int shift;
  int bits;
  unsigned long long drop;
  I2_HOST_DEVICE unsigned long long key(unsigned long long u, unsigned long long v) const { return (u << shift) | v; }
  I2_HOST_DEVICE unsigned long long hi(unsigned long long k) const { return k >> shift; }
  I2_HOST_DEVICE unsigned long long lo(unsigned long long k) const { return k & ((1ull << shift) - 1); }
};

inline int bit_length(unsigned long long x) {
  int b = 0;
  for (; x; x >>= 1) ++b;
  return b;
}

inline KeyBits key_bits(int n) {
  KeyBits k;
  k.shift = bit_length((unsigned long long)n - 1);
  if (k.shift < 1) k.shift = 1;
  k.bits = k.shift + bit_length((unsigned long long)n);
  k.drop = (unsigned long long)n << k.shift;
  return k;
}

}  // namespace i2
