// Prints the order by length of ptx.jl_b200/csrc/attn_sched.cuh, for tests/test_attention_by_length.py.
#include <cstdio>
#include <cstdlib>

#include "attn_sched.cuh"

// usage: attn_sched_dump grid items: each CTA's places in the order, a line per CTA
int main(int argc, char** argv) {
  if (argc != 3) return 1;
  const int grid = std::atoi(argv[1]), items = std::atoi(argv[2]);
  for (int cta = 0; cta < grid; ++cta) {
    for (int v = 0, r; (r = ptxb200::fa_length_rank(cta, v, grid)) < items; ++v) std::printf("%d ", r);
    std::printf("\n");
  }
  return 0;
}
