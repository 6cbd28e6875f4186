// fwd_cols.cuh -- forward column pass of the four-step transforms
#pragma once

#include "device_common.cuh"

namespace b200 {

namespace {

// --------------------------------------------------------------------------
// K1: forward column DFTs with the unpack fused into the load
// --------------------------------------------------------------------------

// columns per 128-thread block: one thread per column, two at n1 = 32
template <int N1>
constexpr unsigned fwd_cols_per_block ()
{
  return N1 == 32 ? 64u : 128u;
}

template <int N1, int KIND>
__global__ void __launch_bounds__ (128, 2)
k_fwd_cols (const InputView in, const float* __restrict__ lut, const uint64_t nkeep,
            const uint64_t part0, const unsigned n2, const float2* __restrict__ tw4,
            float2* __restrict__ scratch, const float* __restrict__ apod)
{
  __shared__ float s_lut[256];
  load_lut (in, lut, s_lut);
  __syncthreads ();
  const unsigned b = blockIdx.y;
  const unsigned c = blockIdx.z;
  const uint64_t N = uint64_t (N1) * n2;
  if constexpr (N1 == 32)
  {
    // Two threads per column (a 32-point DFT in one thread's registers
    // spills): thread h of the pair takes rows 2m + h, a 16-point DFT of
    // them gives E (h = 0) or O (h = 1), thread 1 applies w32^j, and one
    // exchange gives X[j] = E[j] + w32^j O[j] to thread 0 and
    // X[j + 16] = E[j] - w32^j O[j] to thread 1.
    const unsigned h = threadIdx.x & 1;
    const unsigned i2 = blockIdx.x * 64 + (threadIdx.x >> 1);
    const uint64_t t0 = (part0 + b) * nkeep + i2;
    for (unsigned p = 0; p < in.npol; p++)
    {
      float2 v[16];
#pragma unroll
      for (int m = 0; m < 16; m++)
        v[m] = fetch<KIND> (in, s_lut, c, p, t0 + uint64_t (2 * m + h) * n2);
      if (apod)
      {
        // Apodization::operate on the part before the forward FFT (Convolution.C:739-743)
#pragma unroll
        for (int m = 0; m < 16; m++)
        {
          const float w = __ldg (apod + uint64_t (2 * m + h) * n2 + i2);
          v[m] = make_float2 (__fmul_rn (v[m].x, w), __fmul_rn (v[m].y, w));
        }
      }
      RegDFT<16, -1>::run (v);
#pragma unroll
      for (int j = 0; j < 16; j++)
      {
        const float2 mine = h ? tw_mul<32, -1> (j, v[j]) : v[j];
        const float2 other = make_float2 (__shfl_xor_sync (0xffffffffu, mine.x, 1),
                                          __shfl_xor_sync (0xffffffffu, mine.y, 1));
        // thread 0: E + O'; thread 1: E - O' (E is the partner's value)
        v[j] = h ? csub (other, mine) : cadd (mine, other);
      }
      const unsigned k0 = 16 * h;
      float2* dst = scratch + ((uint64_t (b) * in.nchan + c) * in.npol + p) * N + i2;
#pragma unroll
      for (int j = 0; j < 16; j++)
      {
        const unsigned k1 = k0 + j;
        float2 y = v[j];
        // four-step twiddle w_N^{k1 n2} (row k1 of the [n1][n2] table)
        if (k1) y = cmul (y, __ldg (tw4 + uint64_t (k1) * n2 + i2));
        dst[uint64_t (k1) * n2] = y;
      }
    }
    return;
  }
  const unsigned i2 = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t t0 = (part0 + b) * nkeep + i2;
  for (unsigned p = 0; p < in.npol; p++)
  {
    float2 v[N1];
#pragma unroll
    for (int k = 0; k < N1; k++)
      v[k] = fetch<KIND> (in, s_lut, c, p, t0 + uint64_t (k) * n2);
    if (apod)
    {
      // Apodization::operate on the part before the forward FFT (Convolution.C:739-743)
#pragma unroll
      for (int k = 0; k < N1; k++)
      {
        const float w = __ldg (apod + uint64_t (k) * n2 + i2);
        v[k] = make_float2 (__fmul_rn (v[k].x, w), __fmul_rn (v[k].y, w));
      }
    }
    RegDFT<N1, -1>::run (v);
    // four-step twiddle w_N^{k1 n2} (row k1 of the [n1][n2] table; coalesced)
#pragma unroll
    for (int k = 1; k < N1; k++)
      v[k] = cmul (v[k], __ldg (tw4 + uint64_t (k) * n2 + i2));
    float2* dst = scratch + ((uint64_t (b) * in.nchan + c) * in.npol + p) * N + i2;
#pragma unroll
    for (int k = 0; k < N1; k++)
      dst[uint64_t (k) * n2] = v[k];
  }
}

} // namespace

} // namespace b200
