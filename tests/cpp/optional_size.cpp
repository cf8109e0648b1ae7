// OptionalSize (superlinear_gb300/csrc) against a fake of the allocation it guards.
#include <cstdio>

#include "../../superlinear_gb300/csrc/optional_size.h"

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("failed, line %d: %s\n", __LINE__, #x);     \
      return 1;                                               \
    }                                                         \
  } while (0)

int main() {
  sus2g::OptionalSize size;
  size_t have = 0, room = 100;
  int asked = 0;
  auto holds = [&](size_t want) {
    return size.holds(have, want, [&](size_t n) {
      ++asked;
      have = n <= room ? n : 0;  // (a buffer that grows gives up what it had first)
      return n <= room;
    });
  };
  CHECK(holds(0) && asked == 0);
  CHECK(holds(80) && holds(40) && holds(80) && asked == 1);
  CHECK(!holds(120) && !holds(120) && asked == 2 && have == 0);
  room = 200;
  CHECK(!holds(120) && asked == 2);  // the reverse of a forward that went without
  CHECK(holds(90) && asked == 3);    // another layout
  CHECK(holds(150) && holds(120) && asked == 4);
  std::printf("ok\n");
  return 0;
}
