// Prints every permutation code of a shared face and its byte selector:
// "p0 p1 p2 code selector" for all triples of 0..2.
#include <cstdio>

#include "vfr_host.h"

int main() {
  for (uint32_t k = 0; k < 27; ++k) {
    const uint32_t p0 = k / 9, p1 = k / 3 % 3, p2 = k % 3, code = vfr::perm_code(p0, p1, p2);
    std::printf("%u %u %u %u %u\n", p0, p1, p2, code, vfr::perm_selector(code));
  }
  return 0;
}
