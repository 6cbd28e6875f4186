// rows32.cuh -- row transforms with 32 points per thread
#pragma once

#include "device_common.cuh"

namespace b200 {

namespace {

// --------------------------------------------------------------------------
// K2 (persistent): the rows.  Row r holds n2 contiguous values,
// r = ((b*nchan + c)*npol + p)*n1 + k1.
// --------------------------------------------------------------------------

template <int N, int D, int P, bool PI, bool PO>
__device__ __forceinline__ void tpass (const float2* src, float2* dst, float2* v,
                                       const float2* tab)
{
  if constexpr (P < stockham_npass (N))
  {
    constexpr int T = stockham_threads (N);
    constexpr int R = stockham_radix (N, P);
    constexpr int Ns = stockham_ns (N, P);
    StockhamPassT<N, R, T, D, PI, PO>::load (threadIdx.x, src, v);
    __syncthreads ();
    StockhamPassT<N, R, T, D, PI, PO>::compute_store (
        threadIdx.x, Ns, v, dst, P ? tab + pass_table_offset (N, P) : nullptr);
    __syncthreads ();
  }
}

// L2 prefetch of a global range (16-byte aligned, multiple of 16 bytes)
__device__ __forceinline__ void prefetch_l2 (const void* p, unsigned bytes)
{
  asm volatile ("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

template <int N2>
constexpr size_t rows32_smem_bytes ()
{
  return size_t (spad_size (N2) + Row32<N2>::TABN) * sizeof (float2);
}

// CTAs of k_rows32 resident per SM: at 8192 shared memory (one padded row +
// 10 KB of twiddles) and 128 registers per thread allow two; at 4096 three
// (four would cap the registers at 128, where the 4096-point schedule spills).
// A 30 KB pass-2 table shared by a thread's two butterflies (fewer
// instructions) measured slower: 208 KB of shared memory per SM leaves too
// little L1 for the rows' global loads.  So did one CTA per SM running two
// row groups with named barriers on alternate rows of one run (sharing one
// response row in L1): 1.91 against 1.78 ms per C2 step.
template <int N2>
constexpr unsigned rows32_ctas_per_sm ()
{
  return N2 == 8192 ? 2u : 3u;
}

// The convolution row (CONV: forward FFT, x H, inverse FFT; otherwise the
// inverse FFT alone, for the inverse filterbank's stitched spectra) with 32
// points per thread in three radix passes each way (Row32): pass 0 reads the
// row straight from the scratch in natural order, the forward pass 2, the
// response multiply and the inverse pass 0 run in registers, the last pass
// writes the row back in natural order.  One padded row of shared memory per
// CTA, used in place; several CTAs per SM overlap one another's
// barrier-separated phases.  The next row (and its response) is prefetched
// into L2 while this one is transformed.
template <int N2, bool CONV>
__global__ void __launch_bounds__ (Row32<N2>::T, rows32_ctas_per_sm<N2> ())
k_rows32 (float2* scratch, const float2* __restrict__ H, const unsigned n1,
          const unsigned nchan, const unsigned npol, const unsigned nrows, const unsigned inner)
{
  using RS = Row32<N2>;
  constexpr unsigned ROW_BYTES = N2 * sizeof (float2);
  constexpr unsigned CHUNK = 16384;
  extern __shared__ __align__ (16) float2 s_row32[];
  float2* work = s_row32;
  float2* tab1 = work + spad_size (N2);
  float2* th = tab1 + RS::TAB1;
  float2* tl = th + RS::TABH;
  const int tid = threadIdx.x;
  for (int i = tid; i < RS::TABN; i += RS::T) tab1[i] = RS::table_entry (i);

  // Rows are walked with their response row (channel, k1) outermost and the
  // parts and polarisations innermost (inner = parts x polarisations), and
  // each CTA takes a contiguous run of that order: the rows of one response
  // row follow each other on one SM, which keeps the response in its L1
  // (loaded evict-last, the streamed rows evict-first).
  const auto row_of = [=] (unsigned idx, unsigned& hrow) {
    hrow = idx / inner;                             // c * n1 + k1
    const unsigned bp = idx % inner;
    return ((bp / npol) * nchan * n1 + hrow / n1 * n1) * npol + (bp % npol) * n1 + hrow % n1;
  };
  float2 v[32];
  const unsigned run = (nrows + gridDim.x - 1) / gridDim.x;
  const unsigned idx_end = min (nrows, (blockIdx.x + 1) * run);
  for (unsigned idx = blockIdx.x * run; idx < idx_end; idx++)
  {
    unsigned hrow = 0;
    const unsigned row = CONV ? row_of (idx, hrow) : idx;
    float2* grow = scratch + uint64_t (row) * N2;
    const unsigned next = idx + 1;
    if (tid == 0 && next < idx_end)
    {
      unsigned nh = 0;
      const unsigned nrow = CONV ? row_of (next, nh) : next;
      const char* nr = reinterpret_cast<const char*> (scratch + uint64_t (nrow) * N2);
      for (unsigned o = 0; o < ROW_BYTES; o += CHUNK) prefetch_l2 (nr + o, CHUNK);
      if (CONV && nh != hrow)
      {
        const char* hp = reinterpret_cast<const char*> (H + uint64_t (nh) * N2);
        for (unsigned o = 0; o < ROW_BYTES; o += CHUNK) prefetch_l2 (hp + o, CHUNK);
      }
    }
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int r = 0; r < 16; r++) v[16 * b + r] = __ldcs (grow + tid + b * RS::T + r * RS::NS2);
    __syncthreads ();     // the previous row's last shared-memory reads are done
    if constexpr (CONV)
    {
      RS::template p0_compute_store<-1> (tid, v, work);
      __syncthreads ();
      RS::p1_load (tid, work, v);
      __syncthreads ();
      RS::template p1_compute_store<-1> (tid, v, work, tab1);
      __syncthreads ();
      RS::p2_load (tid, work, v);
      __syncthreads ();
      RS::template p2_compute<-1> (tid, v, th, tl);
      // Response::operate (Response.C:662-726): (f_r d_r - f_i d_i, f_i d_r + f_r d_i)
      const float2* h = H + uint64_t (hrow) * N2;
#pragma unroll
      for (int b = 0; b < 2; b++)
#pragma unroll
        for (int r = 0; r < 16; r++)
        {
          const float2 d = v[16 * b + r];
          const float2 f = ldg_evict_last (h + tid + b * RS::T + r * RS::NS2);
          v[16 * b + r] = make_float2 (d.x * f.x - d.y * f.y, d.x * f.y + d.y * f.x);
        }
    }
    RS::template p0_compute_store<+1> (tid, v, work);
    __syncthreads ();
    RS::p1_load (tid, work, v);
    __syncthreads ();
    RS::template p1_compute_store<+1> (tid, v, work, tab1);
    __syncthreads ();
    RS::p2_load (tid, work, v);
    RS::template p2_compute<+1> (tid, v, th, tl);
    RS::p2_store (tid, v, grow);
  }
}

template <int N2, bool CONV>
cudaError_t set_rows_smem ()
{
  return cudaFuncSetAttribute (k_rows32<N2, CONV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int (rows32_smem_bytes<N2> ()));
}

} // namespace

} // namespace b200
