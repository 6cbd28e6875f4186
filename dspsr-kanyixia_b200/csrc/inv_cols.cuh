// inv_cols.cuh -- inverse column transforms shared by the convolution and the
// filterbank with a response
#pragma once

#include "device_common.cuh"

namespace b200 {

namespace {

// One column of an inverse four-step pass: N1 values stride apart, the
// conjugate twiddles tw[k*tw_stride], then the N1-point inverse DFT.
template <int N1>
__device__ __forceinline__ void inv_column (const float2* __restrict__ src, uint64_t stride,
                                            const float2* __restrict__ tw, unsigned tw_stride,
                                            float2* v)
{
#pragma unroll
  for (int k = 0; k < N1; k++)
    v[k] = src[uint64_t (k) * stride];
#pragma unroll
  for (int k = 1; k < N1; k++)
    v[k] = cmulc (v[k], __ldg (tw + uint64_t (k) * tw_stride));
  RegDFT<N1, +1>::run (v);
}

// Two polarisations of 16 or 32 values each do not fit in registers beside
// the DFT's temporaries: the first waits in shared memory (one slot per
// thread, so no barrier) while the second is transformed.
template <int N1, int NPOL>
__host__ __device__ constexpr bool stage_first_pol () { return NPOL == 2 && N1 >= 16; }

} // namespace

} // namespace b200
