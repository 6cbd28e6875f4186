// The bounded mbarrier wait of the row kernels (csrc/tcgen05.cuh) on the GPU:
// a barrier whose phase has completed is seen at once, and one that nothing
// ever completes makes the wait give up within its bound and the kernel end.
// Prints "wait ok=<0|1> ms=<time>" for each.
#include "tcgen05.cuh"

#include <cuda_runtime.h>

#include <cstdio>

__global__ void k_wait (int complete, int* ok, unsigned long long* ns)
{
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) b200::tc::bar_init (&bar, 1);
  __syncthreads ();
  if (complete && threadIdx.x == 0)
    asm volatile ("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b200::tc::saddr (&bar))
                  : "memory");
  __syncthreads ();
  const uint64_t t0 = b200::tc::wall_ns ();
  const bool r = b200::tc::bar_wait (&bar, 0);
  if (threadIdx.x == 0)
  {
    *ok = r;
    *ns = b200::tc::wall_ns () - t0;
  }
}

int main ()
{
  int* ok = nullptr;
  unsigned long long* ns = nullptr;
  if (cudaMallocManaged (&ok, sizeof (*ok)) != cudaSuccess
      || cudaMallocManaged (&ns, sizeof (*ns)) != cudaSuccess)
    return 1;
  for (int complete = 1; complete >= 0; complete--)
  {
    k_wait<<<1, 64>>> (complete, ok, ns);
    if (cudaDeviceSynchronize () != cudaSuccess) return 1;
    printf ("wait ok=%d ms=%.3f\n", *ok, double (*ns) * 1e-6);
  }
  return 0;
}
