// Host-side check of the default chunk of a time-lapse (kernels.cuh, stack_chunk). Usage:
// stack_chunk_check frames plane pageable_out. Built and run by tests/test_stack_chunk.py.
#include "../../sred_b200/csrc/kernels.cuh"

#include <cstdio>
#include <cstdlib>

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  std::printf("%zu\n", sred::stack_chunk(std::atoll(argv[1]), std::atoll(argv[2]), std::atoi(argv[3]) != 0));
  return 0;
}
