// Checks that sorts of different sizes with one build leave every kernel's shared-memory limit alone:
// radix_sort_dispatch (cccl_gb300/csrc/radix_plan.cpp) runs against a driver that records the limits
// and the launches. Threads share a build's kernels, so a limit that follows the call's size could be
// lowered between another call's setting and its launch. Prints one line per failure and exits
// non-zero if any. Built and run by tests/test_smem_limit.py.
#include "radix_plan.h"

#include <cstdint>
#include <cstdio>
#include <map>
#include <set>

#include "abi_common.h"

#include "recording_driver.h"

namespace
{
std::map<CUfunction, std::set<int>> limits; // every value set, by function
int failures = 0;
} // namespace

void limit_set(CUfunction f, int bytes)
{
  limits[f].insert(bytes);
}

void role_launched(const char*) {}

void launched(CUfunction f, unsigned smem)
{
  if (smem > 48 * 1024 && (limits[f].empty() || smem > unsigned(*limits[f].begin())))
  {
    std::printf("a launch of kernel %p takes %u bytes, a call may set less\n", (void*) f, smem);
    ++failures;
  }
}

int main()
{
  using namespace gb300;
  int sorts = 0;
  for (int kb : {1, 2, 4, 8})
  {
    for (int vb : {0, 4, 8})
    {
      limits.clear();
      const RadixPolicy pol = make_radix_policy(kb, vb, KIND_UNSIGNED);
      RadixKernels ks{};
      CUkernel* const slots = reinterpret_cast<CUkernel*>(&ks);
      static_assert(sizeof(RadixKernels) % sizeof(CUkernel) == 0, "nothing but kernels");
      for (size_t i = 0; i < sizeof(RadixKernels) / sizeof(CUkernel); ++i)
      {
        slots[i] = reinterpret_cast<CUkernel>(uintptr_t(i + 1));
      }
      auto sort = [&](uint64_t n, int begin_bit, int end_bit) {
        RadixCall c{};
        // nothing is read or written: addresses only
        for (int i = 0; i < 2; ++i)
        {
          c.keys[i]   = reinterpret_cast<void*>(uintptr_t(1 + i) << 40);
          c.values[i] = vb > 0 ? reinterpret_cast<void*>(uintptr_t(3 + i) << 40) : nullptr;
        }
        size_t bytes         = 0;
        int selector         = 0;
        c.num_items          = n;
        c.begin_bit          = begin_bit;
        c.end_bit            = end_bit;
        c.temp_storage_bytes = &bytes;
        radix_sort_dispatch(pol, ks, c, &selector);
        c.d_temp_storage = reinterpret_cast<void*>(uintptr_t(5) << 40);
        radix_sort_dispatch(pol, ks, c, &selector);
        ++sorts;
      };
      // short sorts of one and more items a thread, longer ones, one digit and all
      for (uint64_t n : {6000ull, 9000ull, 20000ull, 40000ull, 90000ull, 131072ull, 1ull << 20, 1ull << 27})
      {
        sort(n, 0, 8 * kb);
        sort(n, 0, 8);
      }
      for (const auto& f : limits)
      {
        if (f.second.size() != 1)
        {
          std::printf("%d-byte keys, %d-byte values, kernel %p: limits from %d to %d\n", kb, vb, (void*) f.first,
                      *f.second.begin(), *f.second.rbegin());
          ++failures;
        }
        else if (unsigned(*f.second.begin()) > 227u * 1024u)
        {
          std::printf("kernel %p: limit %d\n", (void*) f.first, *f.second.begin());
          ++failures;
        }
      }
    }
  }
  std::printf("%d sorts, %d failures\n", sorts, failures);
  return failures == 0 ? 0 : 1;
}
