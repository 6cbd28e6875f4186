// group_fft.cuh -- shared-memory Stockham transforms run by groups of a block
#pragma once

#include "fft_core.cuh"

namespace b200 {

namespace {

// Stockham FFT of N points run by a group of T = N/16 threads (tid within the
// group) on the group's own shared-memory array; every group of the CTA runs
// the same passes, so the CTA-wide barriers line up.
// Twiddles come from the per-pass tables (pass_table_offset layout) that the
// caller holds in shared memory.
template <int N, int T, int D, int P>
__device__ __forceinline__ void group_fft_pass (float2* s, float2* v, const float2* tab, int tid)
{
  if constexpr (P < stockham_npass (N))
  {
    constexpr int R = stockham_radix (N, P);
    constexpr int Ns = stockham_ns (N, P);
    StockhamPassT<N, R, T, D, true, true>::load (tid, s, v);
    __syncthreads ();
    StockhamPassT<N, R, T, D, true, true>::compute_store (
        tid, Ns, v, s, P ? tab + pass_table_offset (N, P) : nullptr);
    __syncthreads ();
    group_fft_pass<N, T, D, P + 1> (s, v, tab, tid);
  }
}

} // namespace

} // namespace b200
