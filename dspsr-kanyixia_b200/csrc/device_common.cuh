// device_common.cuh -- device code shared by the kernel files: input fetch,
// detection, fold, launch clock
#pragma once

#include "kernels.cuh"
#include "fft_core.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

namespace b200 {

extern std::atomic<uint64_t> g_launches;   // kernels launched since the library was loaded

namespace {

constexpr unsigned FULL = 0xffffffffu;

struct ClockScope
{
  const KernelClock* c;
  int kind;
  cudaStream_t st;
  ClockScope (const KernelClock* c_, int k, cudaStream_t s) : c (c_), kind (k), st (s)
  {
    g_launches++;
    if (c) c->mark (c->self, kind, 0, st);
  }
  ~ClockScope ()
  {
    if (c) c->mark (c->self, kind, 1, st);
  }
};

// --------------------------------------------------------------------------
// input fetch (unpack fused into the load)
// --------------------------------------------------------------------------

template <int KIND>
__device__ __forceinline__ float2 fetch (const InputView& in, const float* s_lut,
                                         unsigned c, unsigned p, uint64_t t)
{
  const void* base = in.main;
  uint64_t span = in.main_span;
  if (t < in.npre)
    base = in.pre, span = in.pre_span;
  else
    t -= in.npre;
  if constexpr (KIND == IN_INT8)
  {
    const uint8_t* b = static_cast<const uint8_t*> (base)
                       + ((t * in.nchan + c) * in.npol + p) * 2;
    const unsigned short w = __ldg (reinterpret_cast<const unsigned short*> (b));
    return make_float2 (s_lut[w & 0xff], s_lut[w >> 8]);
  }
  else if constexpr (KIND == IN_INT16)
  {
    const int16_t* q = static_cast<const int16_t*> (base)
                       + ((t * in.nchan + c) * in.npol + p) * 2;
    const unsigned w = __ldg (reinterpret_cast<const unsigned*> (q));
    short re = short (w & 0xffff), im = short (w >> 16);
    if (in.offset_binary)
    {
      re = short (re ^ 0x8000);
      im = short (im ^ 0x8000);
    }
    // SixteenBitUnpacker.C:69: float(x) + 0.5 (the double 0.5 rounds to float)
    return make_float2 (__fadd_rn (float (re), 0.5f), __fadd_rn (float (im), 0.5f));
  }
  else
  {
    const float2* f = static_cast<const float2*> (base);
    return __ldg (f + (uint64_t (c) * in.npol + p) * span + t);
  }
}

__device__ __forceinline__ void load_lut (const InputView& in, const float* lut, float* s_lut)
{
  if (in.kind == IN_INT8)
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
      s_lut[i] = lut[i];
}

// read-only load kept in L1 ahead of other lines (reused by later rows)
__device__ __forceinline__ float2 ldg_evict_last (const float2* p)
{
  float2 v;
  asm volatile ("ld.global.nc.L1::evict_last.v2.f32 {%0, %1}, [%2];"
                : "=f"(v.x), "=f"(v.y)
                : "l"(p));
  return v;
}

// --------------------------------------------------------------------------
// detection (Detection.C:253-301 Intensity/PPQQ order, cross_detect.ic:38-41,
// stokes_detect.ic:40-43); explicit _rn arithmetic so that no product is
// fused into an FMA and every value rounds as the reference's CPU code does.
// --------------------------------------------------------------------------

__device__ __forceinline__ void detect_values (int state, unsigned npol, float2 p, float2 q,
                                               float* o)
{
  if (state == 0)
  {
    float v = __fmul_rn (p.x, p.x);
    v = __fadd_rn (v, __fmul_rn (p.y, p.y));
    if (npol == 2)
    {
      v = __fadd_rn (v, __fmul_rn (q.x, q.x));
      v = __fadd_rn (v, __fmul_rn (q.y, q.y));
    }
    o[0] = v;
    return;
  }
  const float pp = __fadd_rn (__fmul_rn (p.x, p.x), __fmul_rn (p.y, p.y));
  const float qq = __fadd_rn (__fmul_rn (q.x, q.x), __fmul_rn (q.y, q.y));
  if (state == 1)
  {
    o[0] = pp;
    o[1] = qq;
    return;
  }
  const float re = __fadd_rn (__fmul_rn (p.x, q.x), __fmul_rn (p.y, q.y));
  const float im = __fsub_rn (__fmul_rn (p.x, q.y), __fmul_rn (p.y, q.x));
  if (state == 2)
  {
    o[0] = pp;
    o[1] = qq;
    o[2] = re;
    o[3] = im;
    return;
  }
  o[0] = __fadd_rn (pp, qq);
  o[1] = __fsub_rn (pp, qq);
  o[2] = __fmul_rn (2.0f, re);
  o[3] = __fmul_rn (2.0f, im);
}

// --------------------------------------------------------------------------
// fold
// --------------------------------------------------------------------------

// Index of the plan segment holding sample t (segments are sorted by start).
__device__ __forceinline__ int seg_search (const FoldSegment* __restrict__ segs, int nseg,
                                           uint64_t t)
{
  int lo = 0, hi = nseg - 1;
  while (lo < hi)
  {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg (&segs[mid].start) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Exact bin of plan sample t in segment s (see host_rules.cpp for the algebra):
// y = (m0 + j*dm) * g in integer arithmetic, then one rounded multiply by nbin.
__device__ __forceinline__ unsigned seg_bin (const FoldSegment* __restrict__ segs, int s,
                                             uint64_t t, unsigned nbin)
{
  const uint64_t start = __ldg (&segs[s].start);
  const int64_t m0 = __ldg (&segs[s].m0);
  const int64_t dm = __ldg (&segs[s].dm);
  const double g = __ldg (&segs[s].g);
  const double y = __dmul_rn (double (m0 + int64_t (t - start) * dm), g);
  return __double2uint_rz (__dmul_rn (y, double (nbin)));
}

__device__ __forceinline__ unsigned fold_bin (const FoldSegment* __restrict__ segs, int nseg,
                                              uint64_t t, unsigned nbin)
{
  return seg_bin (segs, seg_search (segs, nseg, t), t, nbin);
}

// Profile columns of a warp whose active lanes hold increasing sample
// indices: one binary search by the first active lane, then each lane steps
// forward over the (few) segment boundaries between it and that lane.  The
// column is the segment's base plus the bin; NO_COLUMN for skipped samples
// and bins outside [0, nbin).  All 32 lanes call this.
constexpr unsigned NO_COLUMN = 0xffffffffu;
__device__ __forceinline__ unsigned warp_fold_bin (const FoldSegment* __restrict__ segs,
                                                   int nseg, bool ok, uint64_t t, unsigned nbin)
{
  const unsigned act = __ballot_sync (FULL, ok);
  if (!act) return NO_COLUMN;
  const int leader = __ffs (act) - 1;
  int s = 0;
  if ((threadIdx.x & 31) == leader) s = seg_search (segs, nseg, t);
  s = __shfl_sync (FULL, s, leader);
  if (!ok) return NO_COLUMN;
  while (s + 1 < nseg && __ldg (&segs[s + 1].start) <= t) s++;
  const unsigned base = __ldg (&segs[s].base);
  const unsigned bin = seg_bin (segs, s, t, nbin);
  return (base == FOLD_SKIP || bin >= nbin) ? NO_COLUMN : base + bin;
}

// Sums of the runs of equal columns in a row (one sample per lane), hm the
// ballot of the lanes that begin a run: a segmented shuffle reduction (a lane
// takes from the lane off further on while that one is in its run, which hm
// tells without asking the other lane), then one atomic per run from its first
// lane, the runs of a row in one instruction.  v is ignored where col is
// NO_COLUMN.
template <int NOUT>
__device__ __forceinline__ void fold_runs (unsigned hm, unsigned col, const float* v, float* prof,
                                           unsigned stride, unsigned* hits)
{
  const int lane = threadIdx.x & 31;
  const unsigned later = (hm >> lane) >> 1;              // heads after this lane
  const int rest = later ? __ffs (later) - 1 : 31 - lane;  // lanes of the run after this one
  float acc[NOUT];
#pragma unroll
  for (int k = 0; k < NOUT; k++) acc[k] = v[k];
  if (hm != FULL)                      // some run is longer than one
  {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
      const bool take = off <= rest;
#pragma unroll
      for (int k = 0; k < NOUT; k++)
      {
        const float o = __shfl_down_sync (FULL, acc[k], off);
        if (take) acc[k] += o;
      }
    }
  }
  if ((hm >> lane & 1) && col != NO_COLUMN)
  {
#pragma unroll
    for (int k = 0; k < NOUT; k++) atomicAdd (prof + uint64_t (k) * stride + col, acc[k]);
    if (hits) atomicAdd (hits + col, unsigned (rest + 1));
  }
}

// Fold of a warp's detected samples where a bin is long (FoldView::long_bins),
// K rows of 32 lanes at a time (a row: the samples the lanes hold for one value
// of a kernel's sample loop).  put() leaves a row in the warp's shared buffer;
// flush() finds the rows that have one column -- most of them -- and has 1 to
// 8 lanes sum each (row, product), 32 values in eight 16-byte loads, one atomic
// each; the others go to fold_runs in one rolled loop.  Against fold_runs for
// every row (5 x NOUT shuffles) C1's inverse columns (n1 = 16) went from 239 to
// 162 us with the rest of the pass; with 11 samples a bin (C2) the detour
// through shared memory is slower, 803 against 664 us at n1 = 8.  Rows of 36 words: the
// row-wise accesses and the 16-byte loads of 8 lanes fall in distinct banks.
template <int NOUT, int K>
struct RowFold
{
  static_assert (NOUT * K <= 32, "a row and product per lane");
  static constexpr int ROWS = K;
  static constexpr int LD = 36;
  static constexpr int WORDS = (NOUT + 1) * K * LD;      // per warp
  float* vals;                                           // [row * NOUT + product][LD]
  unsigned* cols;                                        // [row][LD]
  float* prof;
  unsigned stride;
  unsigned* hits;
  int n = 0;                                             // rows held (warp-uniform)

  __device__ __forceinline__ RowFold (float* warp_buffer, float* p, unsigned st, unsigned* h)
    : vals (warp_buffer), cols (reinterpret_cast<unsigned*> (warp_buffer + NOUT * K * LD)),
      prof (p), stride (st), hits (h)
  {}

  // all 32 lanes, with room for a row (n < K); v is ignored where col is NO_COLUMN
  __device__ __forceinline__ void put (unsigned col, const float* v)
  {
    const int lane = threadIdx.x & 31;
    cols[n * LD + lane] = col;
#pragma unroll
    for (int o = 0; o < NOUT; o++) vals[(n * NOUT + o) * LD + lane] = v[o];
    n++;
  }

  __device__ __forceinline__ void flush ()
  {
    if (n == 0) return;
    const int lane = threadIdx.x & 31;
    unsigned whole = 0;                // rows with one column
#pragma unroll 1
    for (int r = 0; r < n; r++)
    {
      // each lane reads back what it stored
      const unsigned col = cols[r * LD + lane];
      const unsigned prev = __shfl_up_sync (FULL, col, 1);
      const unsigned hm = __ballot_sync (FULL, lane == 0 || prev != col);
      if (hm == 1)
      {
        if (col != NO_COLUMN) whole |= 1u << r;
        continue;
      }
      float v[NOUT];
#pragma unroll
      for (int o = 0; o < NOUT; o++) v[o] = vals[(r * NOUT + o) * LD + lane];
      fold_runs<NOUT> (hm, col, v, prof, stride, hits);
    }
    if (whole)
    {
      __syncwarp ();
      const int rows = n * NOUT;
      const int lg = rows > 16 ? 0 : rows > 8 ? 1 : rows > 4 ? 2 : 3;
      const int sub = lane & ((1 << lg) - 1), len = 32 >> lg;
      const int row = min (lane >> lg, rows - 1);
      const float4* vp = reinterpret_cast<const float4*> (vals + row * LD + sub * len);
      float4 acc = vp[0];
      for (int i = 1; i < len / 4; i++)
      {
        const float4 x = vp[i];
        acc.x += x.x;
        acc.y += x.y;
        acc.z += x.z;
        acc.w += x.w;
      }
      float a = (acc.x + acc.y) + (acc.z + acc.w);
      for (int off = 1; off < (1 << lg); off <<= 1) a += __shfl_xor_sync (FULL, a, off);
      const int k = row / NOUT, o = row % NOUT;
      if (sub == 0 && (lane >> lg) < rows && (whole >> k & 1))
      {
        const unsigned col = cols[k * LD];
        atomicAdd (prof + uint64_t (o) * stride + col, a);
        if (hits && o == 0) atomicAdd (hits + col, 32u);
      }
      __syncwarp ();
    }
    n = 0;
  }
};

// The profile column of sample t of every lane (NO_COLUMN where !ok).
__device__ __forceinline__ unsigned fold_column (const FoldView& fv, bool ok, uint64_t t)
{
  const unsigned col = fv.cols ? (ok ? __ldg (fv.cols + t) : NO_COLUMN)
                               : warp_fold_bin (fv.segs, fv.nseg, ok, t, fv.nbin);
  return col < fv.stride ? col : NO_COLUMN;
}

// One row folded at once.
template <int NOUT>
__device__ __forceinline__ void fold_row (unsigned col, const float* v, float* prof,
                                          unsigned stride, unsigned* hits)
{
  const unsigned prev = __shfl_up_sync (FULL, col, 1);
  const unsigned hm = __ballot_sync (FULL, (threadIdx.x & 31) == 0 || prev != col);
  fold_runs<NOUT> (hm, col, v, prof, stride, hits);
}

// Detects a row and folds it: LONG rows wait in rf (the caller flushes after
// every RowFold::ROWS calls), others are folded at once.  A row with no column
// to go to -- all in the overlap discard -- has nothing to add (the vote is
// warp-uniform).  Callers ask for the columns (fold_column) with the values
// they belong to: loaded here, each row would wait for memory in turn.
template <bool LONG, int NOUT, int K>
__device__ __forceinline__ void detect_row (RowFold<NOUT, K>& rf, int state, unsigned npol,
                                            unsigned col, float2 p, float2 q)
{
  if (!__any_sync (FULL, col != NO_COLUMN)) return;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  detect_values (state, npol, p, q, v);
  if constexpr (LONG)
    rf.put (col, v);
  else
    fold_row<NOUT> (col, v, rf.prof, rf.stride, rf.hits);
}

// The same without a RowFold.
template <int NOUT>
__device__ __forceinline__ void detect_fold (const FoldView& fv, unsigned npol, unsigned col,
                                             float2 p, float2 q, float* prof, unsigned* hits)
{
  if (!__any_sync (FULL, col != NO_COLUMN)) return;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  detect_values (fv.state, npol, p, q, v);
  fold_row<NOUT> (col, v, prof, fv.stride, hits);
}

} // namespace

} // namespace b200
