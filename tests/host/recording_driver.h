// A CUDA driver for radix_sort_dispatch (cccl_gb300/csrc/radix_plan.cpp) on the CPU: every call succeeds, and
// limits and launches go to the including file's limit_set and launched, roles to its role_launched.
#pragma once

#include <cuda.h>

void limit_set(CUfunction f, int bytes);
void launched(CUfunction f, unsigned smem);
void role_launched(const char* role);

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
    limit_set(f, v);
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
void notify_launch(const char* role, int phase, CUstream)
{
  if (phase == 0)
  {
    role_launched(role);
  }
}
} // namespace gb300
