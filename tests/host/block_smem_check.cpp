// Checks that the segmented sort's block classes are launched with shared memory for every form their
// kernels may take (cccl_gb300/csrc/sort_policy.h). Compiled for both block algorithms by
// tests/test_block_smem.py.
#include <cstdio>
#include <initializer_list>

#include "sort_policy.h"

using namespace gb300;

int main()
{
  int failures = 0;
  auto check   = [&](const char* what, int kb, size_t has, size_t needs) {
    if (has < needs)
    {
      std::printf("%s, %d-byte keys: %zu bytes of %zu\n", what, kb, has, needs);
      ++failures;
    }
  };
  for (int kb : {1, 2, 4, 8})
  {
    const int shapes[3][2] = {{seg_block_xs_tpb(kb), seg_block_xs_items(kb)},
                              {seg_block_s_tpb(kb), seg_block_s_items(kb)},
                              {seg_block_l_tpb(kb), seg_block_l_items(kb)}};
    for (const auto& s : shapes)
    {
      check("digit passes", kb, seg_block_smem(kb, s[0], s[1]), block_sort_smem(kb, s[0], s[1]));
      if (seg_block_algo(kb) == SEG_BLOCK_MERGE)
      {
        check("merges", kb, seg_block_smem(kb, s[0], s[1]), block_merge_smem(kb, s[0], s[1]));
      }
    }
  }
  // 512 words a warp, one of padding per 32 (warp_sort.cuh)
  const int tpb = seg_block_s_tpb(4);
  check("groups of warps", 4, seg_block_smem(4, tpb, seg_block_s_items(4)), size_t(tpb / 32) * (512 + 512 / 32) * 4);
  return failures == 0 ? 0 : 1;
}
