// Test-only: compiles the digit arithmetic of the integer router with a host compiler.  Not part of the product library.
#include "../ateniaengine_b200/csrc/router_digits.cuh"

extern "C" int digits_exponent(unsigned largest) { return atenia::digits_x_exponent(largest); }
extern "C" int digits_off(unsigned smallest, int ex) { return atenia::digits_x_off_grid(smallest, ex); }
// smallest value but zeros of n pairs of bf16 patterns, as the kernel's exponent pass finds it
extern "C" unsigned digits_smallest(const unsigned* pairs, int n) {
  auto mins = [](unsigned a, unsigned b) { return (unsigned)(uint16_t)((int16_t)a < (int16_t)b ? a : b); };
  unsigned key = 0x7fffu;
  for (int i = 0; i < n; ++i) {
    const unsigned k = atenia::digits_keys(pairs[i] & 0x7fff7fffu);
    key = mins(key, mins(k & 0xffffu, k >> 16));
  }
  return atenia::digits_of_key(key);
}
extern "C" unsigned digits_x(int X) { return atenia::digits_x_bytes(X); }
extern "C" void digits_w(long long W, signed char* out5, long long* rest) {
  for (int p = 4; p >= 0; --p) out5[p] = atenia::digits_w_next(W);
  *rest = W;
}
extern "C" void digits_levels(const int* A8, long long* p3) {
  int32_t A[8];
  long long p[3];
  for (int i = 0; i < 8; ++i) A[i] = A8[i];
  atenia::digits_fold(A, p);
  for (int i = 0; i < 3; ++i) p3[i] = p[i];
}
