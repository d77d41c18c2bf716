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
#include <vector>

#include "abi_common.h"

namespace
{
std::map<CUfunction, std::set<int>> limits; // every value set, by function
std::map<CUfunction, unsigned> most;        // largest launch, by function
int failures = 0;

void launched(CUfunction f, unsigned smem)
{
  most[f] = most[f] > smem ? most[f] : smem;
  if (smem > 48 * 1024 && (limits[f].empty() || smem > unsigned(*limits[f].begin())))
  {
    std::printf("a launch of kernel %p takes %u bytes, a call may set less\n", (void*) f, smem);
    ++failures;
  }
}
} // namespace

// ---- the driver ----
extern "C" {
CUresult cuGetErrorName(CUresult, const char** s)
{
  *s = "error";
  return CUDA_SUCCESS;
}
CUresult cuKernelGetFunction(CUfunction* f, CUkernel k)
{
  *f = reinterpret_cast<CUfunction>(k);
  return CUDA_SUCCESS;
}
CUresult cuFuncSetAttribute(CUfunction f, CUfunction_attribute a, int v)
{
  if (a == CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES)
  {
    limits[f].insert(v);
  }
  return CUDA_SUCCESS;
}
CUresult cuLaunchKernel(CUfunction f, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned smem,
                        CUstream, void**, void**)
{
  launched(f, smem);
  return CUDA_SUCCESS;
}
CUresult cuLaunchKernelEx(const CUlaunchConfig* c, CUfunction f, void**, void**)
{
  launched(f, c->sharedMemBytes);
  return CUDA_SUCCESS;
}
CUresult cuLaunchCooperativeKernel(CUfunction f, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned,
                                   unsigned smem, CUstream, void**)
{
  launched(f, smem);
  return CUDA_SUCCESS;
}
CUresult cuOccupancyMaxActiveBlocksPerMultiprocessor(int* n, CUfunction, int, size_t)
{
  *n = 1;
  return CUDA_SUCCESS;
}
CUresult cuOccupancyMaxActiveClusters(int* n, CUfunction, const CUlaunchConfig*)
{
  *n = 1;
  return CUDA_SUCCESS;
}
CUresult cuCtxGetDevice(CUdevice* d)
{
  *d = 0;
  return CUDA_SUCCESS;
}
CUresult cuDeviceGetAttribute(int* v, CUdevice_attribute, CUdevice)
{
  *v = 152;
  return CUDA_SUCCESS;
}
CUresult cuMemsetD32Async(CUdeviceptr, unsigned, size_t, CUstream)
{
  return CUDA_SUCCESS;
}
CUresult cuMemcpyAsync(CUdeviceptr, CUdeviceptr, size_t, CUstream)
{
  return CUDA_SUCCESS;
}
}

namespace gb300
{
void notify_launch(const char*, int, CUstream) {}
} // namespace gb300

int main()
{
  using namespace gb300;
  int sorts = 0;
  for (int kb : {1, 2, 4, 8})
  {
    for (int vb : {0, 4, 8})
    {
      limits.clear();
      most.clear();
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
