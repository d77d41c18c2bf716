// finish_choose (cccl_gb300/csrc/sort_policy.h) on the CPU: how many equal keys in the sample of otherwise
// evenly spread ones leave the sort to all digit passes. Built and run by tests/test_finish_copies.py.
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "sort_policy.h"

using namespace gb300;

int main()
{
  int failures = 0;
  for (int kb : {4, 8})
  {
    for (int mode : {PLAN_MODE_SEPARATE, PLAN_MODE_DOUBLE})
    {
      const unsigned long long n = 1ull << 26;
      const uint32_t samples     = finish_sample_items(n);
      const uint32_t cap         = uint32_t(finish_cap(kb, 0, false));
      for (unsigned long long pairs = 0; pairs < 6; ++pairs)
      {
        // S^2 / (2 buckets) pairs of a level; the equal pairs show at every level
        unsigned long long light[MAX_PASSES] = {};
        uint32_t heavy[MAX_PASSES]           = {};
        heavy[0]                             = samples;
        for (int l = 1; l < kb; ++l)
        {
          light[l] = 2 * pairs + (l == 1 ? (unsigned long long) samples * samples >> 16 : l == 2 ? samples * samples >> 24 : 0);
        }
        heavy[kb - 1]       = uint32_t(2 * pairs);
        uint32_t piece      = 0;
        const int digits    = finish_choose(kb, 0u, light, heavy, n, samples, cap, finish_cost(kb, 0), mode, &piece);
        const bool expected = kb == 4 ? pairs < 2 : pairs < 4; // 2 n / S^2 copies of the mean key a pair
        if ((digits != 0) != expected)
        {
          std::printf("%d-byte keys, mode %d, %d pairs: %d digits\n", kb, mode, int(pairs), digits);
          ++failures;
        }
      }
    }
  }
  return failures == 0 ? 0 : 1;
}
