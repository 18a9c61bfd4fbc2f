// Prints what ptx.jl_b200/csrc/gemm_split_plan.h says, for tests/test_gemm_split_plan.py.
#include <cstdio>
#include <initializer_list>

#include "gemm_split_plan.h"

using namespace ptxb200;

int main() {
  const int steps[] = {1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 127, 128, 129, 255, 256, 512, 1024, 1027, 4096};
  for (int bn = 64; bn <= 192; bn += 64)
    for (int split = 1; split <= kMaxParts3; ++split)
      for (int kiters : steps)
        for (int f32 = 0; f32 < 2; ++f32)
          for (int longest : {0, 8, 9, 18, 35, 1024}) {
            if (kiters < split || bn / 16 < split || (bn == 192 && split != 2)) continue;
            const GemmSplitLayout l = gemm_split_layout({bn, split}, kiters, f32 != 0, longest);
            std::printf("layout %d %d %d %d %d %d %d %d %d %d %d %d", bn, split, kiters, f32, longest, l.stages,
                        l.chain_stages, l.fold ? 1 : 0, l.tmem_cols, l.smem_bytes, recv_bytes3(bn, split), stage_k3(bn));
            for (int part = 0; part <= split; ++part) std::printf(" %d", part_begin3(kiters, split, part));
            for (int part = 0; part <= split; ++part) std::printf(" %d", unpack_col3(part_cols3(bn, split), part));
            std::printf("\n");
          }
  for (int tiles : {1, 2, 4, 9, 32, 40, 74, 75, 100})
    for (int kiters : {1, 8, 15, 16, 17, 64, 128, 1024, 4096}) {
      const GemmLine line = gemm_line(148, tiles, 128, 192, kiters);   // a product of one 128x256 tile each
      std::printf("line %d %d %d %d\n", tiles, kiters, line.ctas, line.share);
    }
  // the rule, for products of one row-tile and n columns of 64, on 148 SMs
  const int none[kMaxParts3 + 1] = {0, 148}, b200[kMaxParts3 + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15},
            all[kMaxParts3 + 1] = {0, 148, 74, 49, 37, 29, 24, 21, 18};
  const int* clusters[] = {none, b200, all};
  for (int set = 0; set < 3; ++set)
    for (int rows = 1; rows <= 12; rows += 11)
      for (int n = 1; n <= 300; ++n)
        for (int kiters : {1, 8, 15, 16, 63, 64, 191, 192, 1024, 1600})
          for (int may = 0; may < 2; ++may) {
            GemmSplitPlan p = {0, 0};
            const bool here = gemm_split_rule(148, clusters[set], 1, 128 * rows, 64 * n, kiters, may != 0, &p);
            std::printf("rule %d %d %d %d %d %d %d %d", set, rows, n, kiters, may, here ? 1 : 0, p.bn, p.split);
            std::printf(" %d", here ? clusters[set][p.split] : 0);
            // chains as launch_gemm_split asks for them
            GemmSplitLayout l = {};
            if (here) l = gemm_split_layout(p, kiters, true, may ? gemm_line(148, 1, 128 * rows, 64 * n, kiters).share : 0);
            std::printf(" %d %d\n", l.fold ? 1 : 0, l.tmem_cols);
          }
  return 0;
}
