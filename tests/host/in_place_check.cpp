// Checks that a plain sort whose output is its input runs every digit pass (cccl_gb300/csrc/radix_plan.cpp): with
// an even number of them the first writes the temporary buffer, while a partition by an odd number
// of digits would write over the keys it has still to read. Built and run by tests/test_in_place.py.
#include "radix_plan.h"

#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <set>
#include <string>

#include "abi_common.h"
#include "recording_driver.h"

static std::set<std::string> roles;

void limit_set(CUfunction, int) {}
void launched(CUfunction, unsigned) {}
void role_launched(const char* role)
{
  roles.insert(role);
}

int main()
{
  using namespace gb300;
  int failures = 0;
  for (int kb : {4, 8})
  {
    for (int vb : {0, 4, 8})
    {
      for (int same = 0; same < 4; ++same) // bit 0: the keys' output is their input, bit 1: the values'
      {
        if (vb == 0 && same > 1)
        {
          continue;
        }
        const RadixPolicy pol = make_radix_policy(kb, vb, KIND_UNSIGNED);
        RadixKernels ks{};
        CUkernel* const slots = reinterpret_cast<CUkernel*>(&ks);
        for (size_t i = 0; i < sizeof(RadixKernels) / sizeof(CUkernel); ++i)
        {
          slots[i] = reinterpret_cast<CUkernel>(uintptr_t(i + 1));
        }
        RadixCall c{};
        for (int i = 0; i < 2; ++i)
        {
          c.keys[i]   = reinterpret_cast<void*>(uintptr_t(1 + ((same & 1) ? 0 : i)) << 40);
          c.values[i] = vb > 0 ? reinterpret_cast<void*>(uintptr_t(3 + ((same & 2) ? 0 : i)) << 40) : nullptr;
        }
        size_t bytes         = 0;
        int selector         = 0;
        c.num_items          = 1ull << 27;
        c.end_bit            = 8 * kb;
        c.temp_storage_bytes = &bytes;
        radix_sort_dispatch(pol, ks, c, &selector);
        c.d_temp_storage = reinterpret_cast<void*>(uintptr_t(5) << 40);
        roles.clear();
        radix_sort_dispatch(pol, ks, c, &selector);
        if ((roles.count("finish") != 0) != (same == 0))
        {
          std::printf("%d-byte keys, %d-byte values, same buffers %d: finish launched %d\n", kb, vb, same,
                      int(roles.count("finish")));
          ++failures;
        }
      }
    }
  }
  return failures == 0 ? 0 : 1;
}
