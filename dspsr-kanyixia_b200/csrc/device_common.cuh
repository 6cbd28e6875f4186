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

// All 32 lanes call this together.  Lanes holding consecutive time samples
// with equal bins form runs; each run is summed by a segmented shuffle
// reduction and added to the profile by its first lane with one atomic.
template <int NOUT, bool HITS>
__device__ __forceinline__ void warp_fold_t (bool ok, unsigned bin, const float* v,
                                             float* prof, unsigned nbin, unsigned* hits)
{
  const int lane = threadIdx.x & 31;
  const unsigned key = ok ? bin : 0xffffffffu;
  const unsigned prev = __shfl_up_sync (FULL, key, 1);
  const bool head = (lane == 0) || (prev != key);
  const unsigned hm = __ballot_sync (FULL, head);
  const int rid = __popc (hm & (FULL >> (31 - lane)));
  float acc[NOUT];
#pragma unroll
  for (int k = 0; k < NOUT; k++) acc[k] = ok ? v[k] : 0.0f;
  int cnt = ok ? 1 : 0;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    const int orid = __shfl_down_sync (FULL, rid, off);
    const bool take = (lane + off < 32) && (orid == rid);
#pragma unroll
    for (int k = 0; k < NOUT; k++)
    {
      const float o = __shfl_down_sync (FULL, acc[k], off);
      if (take) acc[k] += o;
    }
    if constexpr (HITS)
    {
      const int oc = __shfl_down_sync (FULL, cnt, off);
      if (take) cnt += oc;
    }
  }
  if (head && ok)
  {
#pragma unroll
    for (int k = 0; k < NOUT; k++)
      atomicAdd (prof + uint64_t (k) * nbin + bin, acc[k]);
    if constexpr (HITS) atomicAdd (hits + bin, unsigned (cnt));
  }
}

// Only the warps that count hits (one channel's) reduce the counts; hits is
// the same pointer in every lane, so the choice is warp-uniform.
template <int NOUT>
__device__ __forceinline__ void warp_fold (bool ok, unsigned bin, const float* v,
                                           float* prof, unsigned nbin, unsigned* hits)
{
  if (hits)
    warp_fold_t<NOUT, true> (ok, bin, v, prof, nbin, hits);
  else
    warp_fold_t<NOUT, false> (ok, bin, v, prof, nbin, hits);
}

template <int NOUT>
__device__ __forceinline__ void emit_fold (const FoldView& fv, unsigned c, unsigned npol, bool ok,
                                           uint64_t t, float2 p, float2 q)
{
  // a warp whose samples all fall in the overlap discard has nothing to add
  // (all 32 lanes are here, so the vote and the return are warp-uniform)
  if (!__any_sync (FULL, ok)) return;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned bin = fv.cols ? (ok ? __ldg (fv.cols + t) : NO_COLUMN)
                         : warp_fold_bin (fv.segs, fv.nseg, ok, t, fv.nbin);
  if (ok)
  {
    detect_values (fv.state, npol, p, q, v);
    ok = bin < fv.stride;
  }
  warp_fold<NOUT> (ok, bin, v, fv.profiles + uint64_t (c) * NOUT * fv.stride, fv.stride,
                   c == 0 ? fv.hits : nullptr);
}

} // namespace

} // namespace b200
