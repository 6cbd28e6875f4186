// rows64.cuh -- 4096-point row transforms with 64 points per thread
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"
#include "tcgen05.cuh"

namespace b200 {

namespace {

// 64-point DFT in registers as 8 x 8: X[k1 + 8 k2] is left in v[8 k1 + k2]
// (r64_out gives the output index of a register)
B200_CE int r64_out (int i) { return (i >> 3) + 8 * (i & 7); }

template <int D>
__device__ __forceinline__ void dft64 (CP* v)
{
#pragma unroll
  for (int n2 = 0; n2 < 8; n2++)
  {
    CP a[8];
#pragma unroll
    for (int n1 = 0; n1 < 8; n1++) a[n1] = v[8 * n1 + n2];
    dft::dft8<D> (a);
#pragma unroll
    for (int k1 = 0; k1 < 8; k1++) v[8 * k1 + n2] = n2 * k1 ? dft::tw64<D> (n2 * k1, a[k1]) : a[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < 8; k1++) dft::dft8<D> (v + 8 * k1);
}

constexpr int R64_N = 4096;             // points per row
constexpr int R64_GROUPS = 4;           // row groups (64 threads each) per block, one block per SM
constexpr int R64_LD = 66;              // exchange row stride (float2)
constexpr int R64_BUF = 64 * R64_LD;    // float2 per group's exchange buffer
constexpr int R64_TW = R64_N / 2;       // twiddle table: w_4096^(q t), q < 32
constexpr size_t R64_SMEM = size_t (R64_TW + R64_GROUPS * R64_BUF) * sizeof (float2);

__device__ __forceinline__ uint32_t r64_saddr (const void* p)
{
  return uint32_t (__cvta_generic_to_shared (p));
}

// the 64 threads of group g
__device__ __forceinline__ void r64_sync (int g)
{
  asm volatile ("bar.sync %0, 64;" ::"r"(g + 1) : "memory");
}

// whether ok holds in every thread of group g
__device__ __forceinline__ bool r64_all (int g, bool ok)
{
  unsigned r;
  asm volatile ("{\n\t.reg .pred p, q;\n\t"
                "setp.ne.u32 p, %1, 0;\n\t"
                "bar.red.and.pred q, %2, 64, p;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(r)
                : "r"(unsigned (ok)), "r"(g + 1)
                : "memory");
  return r != 0;
}

// one thread: copy a row (32 KB, both ends 16-byte aligned) into the group's
// buffer; bar completes when it has landed
__device__ __forceinline__ void r64_load (float2* dst, const float2* src, uint64_t* bar)
{
  constexpr unsigned BYTES = R64_N * sizeof (float2);
  asm volatile ("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(r64_saddr (bar)),
                "r"(BYTES)
                : "memory");
  asm volatile ("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                "[%0], [%1], %2, [%3];" ::"r"(r64_saddr (dst)),
                "l"(src), "r"(BYTES), "r"(r64_saddr (bar))
                : "memory");
}

// K2 for 4096-point rows: forward FFT, x H, inverse FFT (row order and the
// choice of rows per block as in k_rows32).  A row is transformed by two
// warps holding 64 points per thread, 4096 = 64 x 64, so that it crosses
// shared memory once each way where 32 points per thread cross twice and
// where 16 cross twice with twice the twiddles: per 8192 points 4.3 k against
// 8.3 k shared-memory clocks.  Thread t holds x[t + 64 r]; after a 64-point
// DFT over r and the twiddle w^(t q) it hands value q to thread q, whose
// second DFT gives X[q + 64 p] -- the order the inverse starts from.  Four
// independent groups per block (one block per SM: 255 registers a thread)
// meet only at 64-thread barriers and share the twiddle table; the next row
// arrives by a bulk copy into the exchange buffer while the last pass and the
// stores run.  The exchange rows are 66 float2 apart: stores (32 lanes, one
// row) and 16-byte loads (32 rows) are free of bank conflicts.
// Bound by FP32 issue and the latency that eight warps leave open (FMA pipe
// 52 %, shared memory 38 %).  The rows
// of 64 channels x 2 polarisations (C2) went from 1717 us with 32 points per
// thread (k_rows32) to 1300 us.
__global__ void __launch_bounds__ (64 * R64_GROUPS, 1)
k_rows64 (float2* scratch, const float2* __restrict__ H, const unsigned n1, const unsigned nchan,
          const unsigned npol, const unsigned nrows, const unsigned inner, const unsigned run,
          int* err)
{
  extern __shared__ __align__ (16) float2 s_r64[];
  __shared__ uint64_t s_bar[R64_GROUPS];
  float2* tw = s_r64;                              // w_4096^(q t) at [q * 64 + t], q < 32
  const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
  float2* s = s_r64 + R64_TW + g * R64_BUF;
  uint64_t* bar = s_bar + g;
  for (int i = threadIdx.x; i < R64_TW; i += 64 * R64_GROUPS)
  {
    double sn, cs;
    sincospi (-2.0 * double ((i >> 6) * (i & 63)) / double (R64_N), &sn, &cs);
    tw[i] = make_float2 (float (cs), float (sn));
  }
  // the upper half of the twiddles: times w_4096^(32 t), kept in a register (a
  // full table took 1.345 ms where this takes 1.287: the 16 KB are worth more
  // as L1 for the response, which a block's rows share)
  float2 w32;
  {
    double sn, cs;
    sincospi (-2.0 * double (t) / 128.0, &sn, &cs);
    w32 = make_float2 (float (cs), float (sn));
  }
  const auto twiddle = [&] (int q) {
    return q < 32 ? tw[q * 64 + t] : q == 32 ? w32 : cmul (tw[(q - 32) * 64 + t], w32);
  };
  if (t == 0)
    asm volatile ("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(r64_saddr (bar)) : "memory");
  asm volatile ("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads ();
  // rows walked with their response row (channel, k1) outermost; each block
  // takes a contiguous run, its groups alternate rows
  const auto row_of = [=] (unsigned idx, unsigned& hrow) {
    hrow = idx / inner;                             // c * n1 + k1
    const unsigned bp = idx % inner;
    return scratch + uint64_t (((bp / npol) * nchan * n1 + hrow / n1 * n1) * npol
                               + (bp % npol) * n1 + hrow % n1) * R64_N;
  };
  const unsigned first = blockIdx.x * run + g, end = min (nrows, (blockIdx.x + 1) * run);
  unsigned hrow = 0, phase = 0;
  if (t == 0 && first < end) r64_load (s, row_of (first, hrow), bar);
  for (unsigned idx = first; idx < end; idx += R64_GROUPS)
  {
    float2* grow = row_of (idx, hrow);
    unsigned nh = 0;
    const float2* next = idx + R64_GROUPS < end ? row_of (idx + R64_GROUPS, nh) : nullptr;
    if (t == 0 && next)
    {
      for (unsigned o = 0; o < R64_N; o += 2048)
        asm volatile ("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(next + o), "r"(16384u)
                      : "memory");
    }
    if (!r64_all (g, tc::bar_wait (bar, phase)))
    {
      // the copy did not land in time: report, give it a last chance to
      // finish before the block's shared memory goes, and leave
      if (t == 0 && err) *err = 1;
      tc::bar_wait (bar, phase);
      return;
    }
    phase ^= 1;
    CP v[64];
#pragma unroll
    for (int r = 0; r < 64; r++) v[r].z = s[t + 64 * r];
    dft64<-1> (v);
    r64_sync (g);                      // every thread has read the row
#pragma unroll
    for (int i = 0; i < 64; i++)
    {
      const int q = r64_out (i);
      s[q * R64_LD + t] = q ? cmul (v[i].z, twiddle (q)) : v[i].z;
    }
    r64_sync (g);
#pragma unroll
    for (int j = 0; j < 32; j++)
    {
      const float4 x = *reinterpret_cast<const float4*> (s + t * R64_LD + 2 * j);
      v[2 * j].z = make_float2 (x.x, x.y);
      v[2 * j + 1].z = make_float2 (x.z, x.w);
    }
    dft64<-1> (v);
    // Response::operate (Response.C:662-726): (f_r d_r - f_i d_i, f_i d_r + f_r d_i)
    CP u[64];
    const float2* h = H + uint64_t (hrow) * R64_N + t;
#pragma unroll
    for (int i = 0; i < 64; i++)
    {
      const int p = r64_out (i);
      u[p].z = cmul (v[i].z, ldg_evict_last (h + 64 * p));
    }
    dft64<+1> (u);
    r64_sync (g);                      // every thread has read the forward exchange
#pragma unroll
    for (int i = 0; i < 64; i++)
    {
      const int q = r64_out (i);
      s[q * R64_LD + t] = q ? cmulc (u[i].z, twiddle (q)) : u[i].z;
    }
    r64_sync (g);
#pragma unroll
    for (int j = 0; j < 32; j++)
    {
      const float4 x = *reinterpret_cast<const float4*> (s + t * R64_LD + 2 * j);
      v[2 * j].z = make_float2 (x.x, x.y);
      v[2 * j + 1].z = make_float2 (x.z, x.w);
    }
    // the buffer is free once every thread has read it: the next row comes in
    asm volatile ("fence.proxy.async.shared::cta;" ::: "memory");
    r64_sync (g);
    if (t == 0 && next) r64_load (s, next, bar);
    dft64<+1> (v);
#pragma unroll
    for (int i = 0; i < 64; i++) grow[t + 64 * r64_out (i)] = v[i].z;
  }
}

// the persistent grid: one block per SM, or as many as have four rows
inline void launch_rows64 (unsigned nrows, float2* scratch, const float2* H, unsigned n1,
                           unsigned nchan, unsigned npol, int nsm, int* err, cudaStream_t st)
{
  const unsigned grid = std::min<unsigned> ((nrows + R64_GROUPS - 1) / R64_GROUPS, unsigned (nsm));
  const unsigned per = (nrows + grid * R64_GROUPS - 1) / (grid * R64_GROUPS);
  k_rows64<<<grid, 64 * R64_GROUPS, R64_SMEM, st>>> (scratch, H, n1, nchan, npol, nrows,
                                                     nrows / (n1 * nchan), per * R64_GROUPS, err);
}

} // namespace

} // namespace b200
