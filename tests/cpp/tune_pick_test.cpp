// pick_fastest (libbi_b200/csrc/tune_pick.h) with fake timings.
#include "../../libbi_b200/csrc/tune_pick.h"

#include <cmath>
#include <cstdio>

#define CHECK(...)                                \
  do {                                            \
    if (!(__VA_ARGS__)) {                               \
      std::printf("line %d: %s\n", __LINE__, #__VA_ARGS__); \
      return 1;                                   \
    }                                             \
  } while (0)

int main() {
  float med[6];
  int best = 7;
  int calls[6] = {};
  {  // the smallest median wins, not the smallest first time
    const float ms[3][3] = {{1.0f, 3.0f, 3.0f}, {1.1f, 1.2f, 1.2f}, {2.0f, 0.1f, 0.1f}};
    auto f = [&](int k, float* t) { *t = ms[k][calls[k]++]; return 0; };
    CHECK(bpf::pick_fastest<6, 3>(3, 1.25f, f, med, &best) == 0 && best == 1);
    // one that the first round shows far from the best is timed once
    CHECK(calls[0] == 3 && calls[1] == 3 && calls[2] == 1 && med[2] == 2.0f && med[1] == 1.2f);
  }
  {  // candidates that cannot be launched drop out, whichever they are
    for (int bad = 0; bad < 4; ++bad) {
      auto f = [&](int k, float* t) { *t = 1.0f + k; return k == bad ? 5 : 0; };
      CHECK(bpf::pick_fastest<6, 3>(4, 10.0f, f, med, &best) == 0 && best == (bad == 0 ? 1 : 0));
      CHECK(std::isinf(med[bad]));
    }
  }
  {  // also one that fails in a later round, although it was the fastest
    int n = 0;
    auto f = [&](int k, float* t) { *t = 1.0f + k; return k == 0 && n++ == 1 ? 5 : 0; };
    CHECK(bpf::pick_fastest<6, 3>(3, 10.0f, f, med, &best) == 0 && best == 1 && std::isinf(med[0]));
  }
  {  // and when the others had dropped out as slow by then
    int n = 0;
    auto f = [&](int k, float* t) { *t = k == 0 ? 1.0f : 2.0f + k; return k == 0 && n++ == 1 ? 5 : 0; };
    CHECK(bpf::pick_fastest<6, 3>(3, 1.25f, f, med, &best) == 0 && best == 1);
  }
  {  // none left: the error
    auto f = [&](int, float*) { return 5; };
    CHECK(bpf::pick_fastest<6, 3>(4, 1.25f, f, med, &best) == 5 && best == -1);
  }
  std::puts("ok");
  return 0;
}
