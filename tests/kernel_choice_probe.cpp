// Test-only: compiles the kernel-choice rules with a host compiler.  Not part of the product library.
#include "../ateniaengine_b200/csrc/kernel_choice.cuh"

extern "C" int choice_i8_decode(int rows, int experts, int d, int F, int shared) {
  return atenia::i8_decode_pays(rows, experts, d, F, shared != 0);
}
extern "C" int choice_bf16(int rows, int groups, int k, int beside) {
  return atenia::bf16_product_kernel(rows, groups, k, beside != 0);
}
extern "C" int choice_shared_rides(int tokens, int tile, int d, int Fs) {
  return atenia::shared_rides_along(tokens, tile, d, Fs);
}
extern "C" int choice_router_i8(int tokens, int d, int experts) { return atenia::router_i8_pays(tokens, d, experts); }
extern "C" int choice_pair_tokens(int rows, int groups, int f_tiles) { return atenia::pair_tokens_of(rows, groups, f_tiles); }
