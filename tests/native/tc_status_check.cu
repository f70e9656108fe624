// Host-side check of the error that each status word of the tensor-core kernel becomes.
// Built and run by tests/test_tc_status.py.
#include "../../sred_b200/csrc/common.cuh"

#include <cstdio>

int main() {
  for (int s = 1; s <= 5; s++) {
    const char* msg = nullptr;
    const sred_status e = sred::tc_status_error(s, &msg);
    std::printf("%d %d %s\n", s, (int)e, msg);
  }
  return 0;
}
