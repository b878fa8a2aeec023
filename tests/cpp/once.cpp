// build_once: a first build that fails in either step leaves nothing behind,
// and the next call builds again.
#include <cstdio>

#include "../../chronusq_public_b200/csrc/cqf_once.hpp"

int main() {
  int store[4] = {0, 0, 0, 0}, made = 0, dropped = 0, failMake = 1, failFill = 1;
  int* slot = nullptr;
  auto call = [&] {
    return cqf::build_once(
        slot, 0,
        [&](int** p) {
          if (failMake) return 2;
          *p = &store[made++];
          return 0;
        },
        [&](int* p) {
          if (failFill) return 3;
          *p = 7;
          return 0;
        },
        [&](int* p) { dropped += p == &store[made - 1]; });
  };
  bool ok = call() == 2 && !slot && !dropped;         // no memory
  failMake = 0;
  ok = ok && call() == 3 && !slot && dropped == 1;    // nothing written: not published
  failFill = 0;
  ok = ok && call() == 0 && slot == &store[1] && *slot == 7;
  ok = ok && call() == 0 && made == 2;                // there already
  std::printf("%s\n", ok ? "ok" : "wrong");
  return ok ? 0 : 1;
}
