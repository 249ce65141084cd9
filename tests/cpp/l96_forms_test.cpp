// The choice of the Lorenz '96 transition's form (libbi_b200/csrc/l96_forms.h).
#include "../../libbi_b200/csrc/l96_forms.h"

#include <cstdio>

#define CHECK(c)                                             \
  do {                                                       \
    if (!(c)) {                                              \
      std::printf("line %d: %s, d = %d\n", __LINE__, #c, d); \
      return 1;                                              \
    }                                                        \
  } while (0)

int main() {
  const int dims[] = {4, 8, 16, 32, 40};
  for (int d : dims)
    for (int blocks = 1; blocks < 10000; ++blocks) {
      const int f32 = bpf::l96_pair_blocks(d, 4, blocks), f64 = bpf::l96_pair_blocks(d, 8, blocks);
      if (d == 4) {
        CHECK(f32 == 0 && f64 == 0);
        continue;
      }
      CHECK(f32 == (blocks <= 296 ? 2 : blocks <= 444 ? 3 : 0));
      // few components in FP64: two threads only while their blocks are all
      // resident; many: at every size (the one-thread form is not compiled)
      CHECK(f64 == (d >= 32 || blocks <= 296 ? 2 : 0));
    }
  std::puts("ok");
  return 0;
}
