// A step due once per device runs again on a second device, after a failure, and
// on every call past the devices it can remember.
#include <cstdio>

#include "../../calaman_g_b200/csrc/once_per_device.hpp"

enum Status { kOk = 0, kFailed = 7 };

#define CHECK(c)                                    \
  do {                                              \
    if (!(c)) {                                     \
      std::printf("line %d: %s\n", __LINE__, #c);   \
      return 1;                                     \
    }                                               \
  } while (0)

int main() {
  static clm::OncePerDevice once;
  int runs = 0;
  Status answer = kOk;
  auto step = [&] {
    ++runs;
    return answer;
  };
  CHECK(once.run(0, step) == kOk && runs == 1);
  CHECK(once.run(0, step) == kOk && runs == 1);
  CHECK(once.run(1, step) == kOk && runs == 2);
  CHECK(once.run(63, step) == kOk && runs == 3);
  CHECK(once.run(1, step) == kOk && once.run(63, step) == kOk && once.run(0, step) == kOk && runs == 3);
  answer = kFailed;
  CHECK(once.run(2, step) == kFailed && runs == 4);
  answer = kOk;
  CHECK(once.run(2, step) == kOk && runs == 5);
  CHECK(once.run(2, step) == kOk && runs == 5);
  CHECK(once.run(64, step) == kOk && once.run(64, step) == kOk && runs == 7);
  std::printf("once_per_device_check ok\n");
  return 0;
}
