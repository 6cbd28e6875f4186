// fwd_cols_pair.cuh -- forward column pass for two polarisations at a time
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"

namespace b200 {

namespace {

// Raw dual-polarisation sample of one channel: 4 bytes (int8), 8 (int16) or
// two float2 in their own rows.
template <int KIND> struct RawPair { using T = unsigned; };
template <> struct RawPair<IN_INT16> { using T = uint2; };
template <> struct RawPair<IN_FLOAT> { using T = float4; };

struct UnpackPair
{
  const float* lut;      // shared-memory table (int8 that is not affine)
  float scale;           // AFFINE: value (x + 0.5) * scale
  unsigned flip;         // int16: xor that leaves the sample offset by 32768
};

// Both polarisations of a raw sample, bit for bit what fetch() gives.  The
// integer forms set the sample's bits under 2^23's exponent (exact), take the
// offset off (exact) and, for int8, form x * scale + 0.5 * scale in one fma:
// both x and 0.5 * scale are exact, so it rounds as (x + 0.5) * scale does.
template <int KIND, bool AFFINE>
__device__ __forceinline__ C2 unpack_pair (typename RawPair<KIND>::T w, const UnpackPair& u)
{
  if constexpr (KIND == IN_INT8 && AFFINE)
  {
    w ^= 0x80808080u;
    float2 re = make_float2 (__uint_as_float (__byte_perm (w, 0x4b000000u, 0x7540)),
                             __uint_as_float (__byte_perm (w, 0x4b000000u, 0x7542)));
    float2 im = make_float2 (__uint_as_float (__byte_perm (w, 0x4b000000u, 0x7541)),
                             __uint_as_float (__byte_perm (w, 0x4b000000u, 0x7543)));
    const float2 off = dft::dup (-8388736.f);          // 2^23 + 128
    const float2 sc = dft::dup (u.scale), half = dft::dup (0.5f * u.scale);
    return {__ffma2_rn (__fadd2_rn (re, off), sc, half), __ffma2_rn (__fadd2_rn (im, off), sc, half)};
  }
  else if constexpr (KIND == IN_INT8)
    return {make_float2 (u.lut[w & 0xff], u.lut[(w >> 16) & 0xff]),
            make_float2 (u.lut[(w >> 8) & 0xff], u.lut[w >> 24])};
  else if constexpr (KIND == IN_INT16)
  {
    const unsigned a = w.x ^ u.flip, b = w.y ^ u.flip;
    const float2 re = make_float2 (__uint_as_float (__byte_perm (a, 0x4b000000u, 0x7610)),
                                   __uint_as_float (__byte_perm (b, 0x4b000000u, 0x7610)));
    const float2 im = make_float2 (__uint_as_float (__byte_perm (a, 0x4b000000u, 0x7632)),
                                   __uint_as_float (__byte_perm (b, 0x4b000000u, 0x7632)));
    const float2 off = dft::dup (-8421376.f);          // 2^23 + 32768
    const float2 half = dft::dup (0.5f);
    return {__fadd2_rn (__fadd2_rn (re, off), half), __fadd2_rn (__fadd2_rn (im, off), half)};
  }
  else
    return {make_float2 (w.x, w.z), make_float2 (w.y, w.w)};
}

template <int KIND>
__device__ __forceinline__ typename RawPair<KIND>::T load_pair (const void* base, uint64_t idx,
                                                                 uint64_t span)
{
  if constexpr (KIND == IN_FLOAT)
  {
    const float2* f = static_cast<const float2*> (base) + idx;
    const float2 p = __ldg (f), q = __ldg (f + span);
    return make_float4 (p.x, p.y, q.x, q.y);
  }
  else
    return __ldg (static_cast<const typename RawPair<KIND>::T*> (base) + idx);
}

// TFPD channels per tile of the transposing load, and the row stride of its
// buffer (words): a warp stores 4 columns x 8 channels and loads 32 columns
// of one channel, both in distinct banks
constexpr int FWP_CH = 8, FWP_LD = 36;
// the same for tiles of 16 columns (a half-warp loads one channel's)
constexpr int FWP32_LD = 20;

template <int N1, int KIND, bool TILE>
constexpr size_t fwp_smem ()
{
  return TILE ? size_t (N1) * FWP_CH * FWP_LD * sizeof (typename RawPair<KIND>::T) : 0;
}

// Threads per block: 128 columns of one channel, or with TILE 32 columns of 8.
template <bool TILE> B200_CE int fwp_threads () { return TILE ? 256 : 128; }
// resident blocks per SM that the registers are sized for
template <int N1, bool TILE> B200_CE int fwp_blocks () { return N1 == 16 ? (TILE ? 2 : 3) : TILE ? 3 : 6; }

// K1 for two polarisations and n1 = 2 .. 16: a thread holds one column of both
// polarisations (C2), one load per raw sample, one twiddle for both.  Blocks
// loop over the parts b = blockIdx.y, + gridDim.y, ... with their twiddles
// kept in registers.  TILE (TFPD integers, a multiple of eight channels): 32
// columns of eight channels are loaded in address order -- a whole 32-byte
// sector (int8) per time sample -- and transposed through shared memory;
// thread by thread each sector would be fetched once per channel.
// Bound by HBM (4 or 8 B in, 16 B out per point of both polarisations) and by
// issue.  Against a thread per polarisation: 10.5 M samples of one channel at
// n1 = 16 172 us before, 108 us now (119 us at n1 = 32, where 2^17 points go
// with 4096-point rows); 32 channels at n1 = 2 180 and 82 us;
// 2^18-point transforms of int16 at n1 = 32 (below) 76 and 46 us.
template <int N1, int KIND, bool AFFINE, bool TILE>
__global__ void __launch_bounds__ (fwp_threads<TILE> (), fwp_blocks<N1, TILE> ())
k_fwd_cols_pair (const InputView in, const float* __restrict__ lut, const uint64_t nkeep,
                 const uint64_t part0, const unsigned nbatch, const unsigned n2,
                 const float2* __restrict__ tw4, float2* __restrict__ scratch,
                 const float* __restrict__ apod)
{
  using Raw = typename RawPair<KIND>::T;
  __shared__ float s_lut[KIND == IN_INT8 && !AFFINE ? 256 : 1];
  extern __shared__ __align__ (16) unsigned char s_fwp[];
  Raw* tile = reinterpret_cast<Raw*> (s_fwp);
  if (KIND == IN_INT8 && !AFFINE)
  {
    load_lut (in, lut, s_lut);
    __syncthreads ();
  }
  const UnpackPair u {s_lut, in.lut_scale, in.offset_binary ? 0u : 0x80008000u};
  const unsigned c0 = TILE ? blockIdx.z * FWP_CH : blockIdx.z;
  const unsigned c = TILE ? c0 + threadIdx.x / 32 : c0;
  const unsigned i0 = blockIdx.x * (TILE ? 32 : 128);
  const unsigned i2 = i0 + (TILE ? threadIdx.x % 32 : threadIdx.x);
  const uint64_t N = uint64_t (N1) * n2;
  // samples per time step of the address space (FPT: one row per polarisation)
  const uint64_t step = KIND == IN_FLOAT ? 1 : in.nchan;
  float2 w[N1];
#pragma unroll
  for (int k = 1; k < N1; k++) w[k] = __ldg (tw4 + uint64_t (k) * n2 + i2);
  for (unsigned b = blockIdx.y; b < nbatch; b += gridDim.y)
  {
    // the block's window lies in one segment of the input (the carried prefix
    // or the main block) except where a part straddles the prefix's end
    const uint64_t ta = (part0 + b) * nkeep + i0;
    const bool in_pre = ta < in.npre;
    const bool one = !in_pre || ta + uint64_t (N1 - 1) * n2 + 127 < in.npre;
    const void* seg = in_pre ? in.pre : in.main;
    const uint64_t span = in_pre ? in.pre_span : in.main_span;
    const uint64_t ts = in_pre ? ta : ta - in.npre;
    // address of time t (from ta) of channel ch
    const auto at = [&] (uint64_t t, unsigned ch) -> Raw {
      const void* s = seg;
      uint64_t sp = span, tt = ts + t;
      if (!one && ta + t >= in.npre)
      {
        s = in.main;
        sp = in.main_span;
        tt = ta + t - in.npre;
      }
      return load_pair<KIND> (s, KIND == IN_FLOAT ? uint64_t (ch) * 2 * sp + tt : tt * step + ch, sp);
    };
    Raw raw[N1];
    if constexpr (TILE)
    {
      const unsigned col = threadIdx.x / FWP_CH, ch = threadIdx.x % FWP_CH;
#pragma unroll
      for (int k = 0; k < N1; k++) raw[k] = at (uint64_t (k) * n2 + col, c0 + ch);
      __syncthreads ();                // the previous part's reads are done
#pragma unroll
      for (int k = 0; k < N1; k++) tile[(k * FWP_CH + ch) * FWP_LD + col] = raw[k];
      __syncthreads ();
#pragma unroll
      for (int k = 0; k < N1; k++)
        raw[k] = tile[(k * FWP_CH + threadIdx.x / 32) * FWP_LD + threadIdx.x % 32];
    }
    else
    {
#pragma unroll
      for (int k = 0; k < N1; k++) raw[k] = at (uint64_t (k) * n2 + threadIdx.x, c);
    }
    C2 v[N1];
#pragma unroll
    for (int k = 0; k < N1; k++) v[k] = unpack_pair<KIND, AFFINE> (raw[k], u);
    if (apod)
    {
      // Apodization::operate on the part before the forward FFT (Convolution.C:739-743)
#pragma unroll
      for (int k = 0; k < N1; k++)
      {
        const float2 a = dft::dup (__ldg (apod + uint64_t (k) * n2 + i2));
        v[k].re = __fmul2_rn (v[k].re, a);
        v[k].im = __fmul2_rn (v[k].im, a);
      }
    }
    dft::run<N1, -1> (v);
    // four-step twiddle w_N^{k1 n2}, in scalars: the products land in the
    // (re, im) pairs that are stored
    float2* d0 = scratch + (uint64_t (b) * in.nchan + c) * 2 * N + i2;
#pragma unroll
    for (int k = 0; k < N1; k++)
    {
      const float2 p = make_float2 (v[k].re.x, v[k].im.x), q = make_float2 (v[k].re.y, v[k].im.y);
      d0[uint64_t (k) * n2] = k ? cmul (p, w[k]) : p;
      d0[N + uint64_t (k) * n2] = k ? cmul (q, w[k]) : q;
    }
  }
}

// Threads per block of the n1 = 32 pass: 64 columns of one channel, or with
// TILE 16 columns of 8 channels, two threads per column.
template <bool TILE> B200_CE int fwp32_threads () { return TILE ? 256 : 128; }
template <int KIND, bool TILE>
constexpr size_t fwp32_smem ()
{
  return size_t (16) * fwp32_threads<TILE> () * sizeof (float4)
         + (TILE ? 32 * FWP_CH * FWP32_LD * sizeof (typename RawPair<KIND>::T) : 0);
}

// The same for n1 = 32: two threads per column, thread h with rows 2m + h (16
// points of both polarisations in registers; 32 spill).  They exchange
// through shared memory -- E, and w32^j O already turned -- and each forms
// X[j] = E[j] + w32^j O[j] and X[j + 16] = E[j] - w32^j O[j] for half the j.
template <int KIND, bool AFFINE, bool TILE>
__global__ void __launch_bounds__ (fwp32_threads<TILE> (), TILE ? 2 : 4)
k_fwd_cols_pair32 (const InputView in, const float* __restrict__ lut, const uint64_t nkeep,
                   const uint64_t part0, const unsigned nbatch, const unsigned n2,
                   const float2* __restrict__ tw4, float2* __restrict__ scratch,
                   const float* __restrict__ apod)
{
  using Raw = typename RawPair<KIND>::T;
  constexpr int T = fwp32_threads<TILE> (), P = T / 2;     // (column, channel) pairs of the block
  constexpr int COLS = TILE ? 16 : 64;
  __shared__ float s_lut[KIND == IN_INT8 && !AFFINE ? 256 : 1];
  extern __shared__ __align__ (16) unsigned char s_fwp[];
  float4* s_x = reinterpret_cast<float4*> (s_fwp);         // [half][j][pair]
  Raw* tile = reinterpret_cast<Raw*> (s_fwp + size_t (16) * T * sizeof (float4));
  if (KIND == IN_INT8 && !AFFINE)
  {
    load_lut (in, lut, s_lut);
    __syncthreads ();
  }
  const UnpackPair u {s_lut, in.lut_scale, in.offset_binary ? 0u : 0x80008000u};
  const unsigned pr = threadIdx.x % P, h = threadIdx.x / P;
  const unsigned c0 = TILE ? blockIdx.z * FWP_CH : blockIdx.z, c = c0 + pr / COLS;
  const unsigned i0 = blockIdx.x * COLS, i2 = i0 + pr % COLS;
  const uint64_t N = 32ull * n2;
  const uint64_t step = KIND == IN_FLOAT ? 1 : in.nchan;
  for (unsigned b = blockIdx.y; b < nbatch; b += gridDim.y)
  {
    const uint64_t ta = (part0 + b) * nkeep + i0;
    const auto at = [&] (uint64_t t, unsigned ch) -> Raw {
      t += ta;
      const bool pre = t < in.npre;
      const uint64_t sp = pre ? in.pre_span : in.main_span, tt = pre ? t : t - in.npre;
      return load_pair<KIND> (pre ? in.pre : in.main,
                              KIND == IN_FLOAT ? uint64_t (ch) * 2 * sp + tt : tt * step + ch, sp);
    };
    C2 v[16];
    {
      Raw raw[16];
      if constexpr (TILE)
      {
        // 16 columns x 8 channels of every row, in address order
        const unsigned ch = threadIdx.x % FWP_CH, col = threadIdx.x / FWP_CH % COLS;
        const unsigned odd = threadIdx.x / (FWP_CH * COLS);
#pragma unroll
        for (int m = 0; m < 16; m++) raw[m] = at (uint64_t (2 * m + odd) * n2 + col, c0 + ch);
#pragma unroll
        for (int m = 0; m < 16; m++)
          tile[((2 * m + odd) * FWP_CH + ch) * FWP32_LD + col] = raw[m];
        __syncthreads ();
#pragma unroll
        for (int m = 0; m < 16; m++)
          raw[m] = tile[((2 * m + h) * FWP_CH + pr / COLS) * FWP32_LD + pr % COLS];
      }
      else
      {
#pragma unroll
        for (int m = 0; m < 16; m++) raw[m] = at (uint64_t (2 * m + h) * n2 + pr, c);
      }
#pragma unroll
      for (int m = 0; m < 16; m++) v[m] = unpack_pair<KIND, AFFINE> (raw[m], u);
    }
    if (apod)
    {
      // Apodization::operate on the part before the forward FFT (Convolution.C:739-743)
#pragma unroll
      for (int m = 0; m < 16; m++)
      {
        const float2 a = dft::dup (__ldg (apod + uint64_t (2 * m + h) * n2 + i2));
        v[m].re = __fmul2_rn (v[m].re, a);
        v[m].im = __fmul2_rn (v[m].im, a);
      }
    }
    dft::run<16, -1> (v);
    if (h)
    {
#pragma unroll
      for (int j = 1; j < 16; j++) v[j] = dft::tw64<-1> (2 * j, v[j]);
    }
    __syncthreads ();                  // the last part's reads are done
#pragma unroll
    for (int j = 0; j < 16; j++)
      s_x[(h * 16 + j) * P + pr] = make_float4 (v[j].re.x, v[j].re.y, v[j].im.x, v[j].im.y);
    __syncthreads ();
    float2* d0 = scratch + (uint64_t (b) * in.nchan + c) * 2 * N + i2;
#pragma unroll
    for (int m = 0; m < 8; m++)
    {
      const unsigned j = 8 * h + m;
      const float4 a = s_x[j * P + pr], o = s_x[(16 + j) * P + pr];
      const C2 e = {make_float2 (a.x, a.y), make_float2 (a.z, a.w)};
      const C2 f = {make_float2 (o.x, o.y), make_float2 (o.z, o.w)};
      const C2 x[2] = {dft::add (e, f), dft::sub (e, f)};
#pragma unroll
      for (int s = 0; s < 2; s++)
      {
        // four-step twiddle w_N^{k1 n2} (row k1 of the [n1][n2] table)
        const unsigned k1 = j + 16 * s;
        const float2 w = k1 ? __ldg (tw4 + uint64_t (k1) * n2 + i2) : make_float2 (1.f, 0.f);
        d0[uint64_t (k1) * n2] = cmul (make_float2 (x[s].re.x, x[s].im.x), w);
        d0[N + uint64_t (k1) * n2] = cmul (make_float2 (x[s].re.y, x[s].im.y), w);
      }
    }
  }
}

template <int N1, int KIND, bool AFFINE, bool TILE>
void launch_fwd_pair_t (const InputView& in, const float* lut, uint64_t nkeep, uint64_t part0,
                        unsigned nbatch, unsigned n2, const float2* tw4, float2* scratch,
                        const float* apod, int nsm, cudaStream_t st)
{
  if constexpr (N1 == 32)
  {
    const unsigned gx = n2 / (TILE ? 16 : 64), gz = TILE ? in.nchan / FWP_CH : in.nchan;
    const unsigned want = std::max (1u, (TILE ? 16 : 32) * unsigned (nsm) / std::max (1u, gx * gz));
    auto kern = k_fwd_cols_pair32<KIND, AFFINE, TILE>;
    constexpr size_t smem = fwp32_smem<KIND, TILE> ();
    if (TILE)
      cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
    kern<<<dim3 (gx, std::min (nbatch, want), gz), fwp32_threads<TILE> (), smem, st>>> (
        in, lut, nkeep, part0, nbatch, n2, tw4, scratch, apod);
    return;
  }
  else
  {
  constexpr int T = fwp_threads<TILE> ();
  const unsigned gx = n2 / (TILE ? 32 : 128), gz = TILE ? in.nchan / FWP_CH : in.nchan;
  // about eight blocks of work per resident block, then parts per block
  const unsigned resident = unsigned (nsm) * fwp_blocks<N1, TILE> ();
  const unsigned want = std::max (1u, 8 * resident / std::max (1u, gx * gz));
  k_fwd_cols_pair<N1, KIND, AFFINE, TILE><<<dim3 (gx, std::min (nbatch, want), gz), T,
                                            fwp_smem<N1, KIND, TILE> (), st>>> (
      in, lut, nkeep, part0, nbatch, n2, tw4, scratch, apod);
  }
}

// Whether the input's samples can be read whole: both polarisations in one
// aligned word (a caller's block may start at any sample of any buffer).
inline bool fwd_pair_aligned (const InputView& in)
{
  const uintptr_t a = reinterpret_cast<uintptr_t> (in.main)
                      | (in.npre ? reinterpret_cast<uintptr_t> (in.pre) : 0);
  return a % (in.kind == IN_INT8 ? 4 : 8) == 0;
}

// Two polarisations, aligned (fwd_pair_aligned).  A multiple of eight TFPD
// channels takes the transposing load; an affine 8-bit table is computed
// instead of looked up.
template <int N1>
void launch_fwd_pair (const InputView& in, const float* lut, uint64_t nkeep, uint64_t part0,
                      unsigned nbatch, unsigned n2, const float2* tw4, float2* scratch,
                      const float* apod, int nsm, cudaStream_t st)
{
  const bool tile = in.nchan % FWP_CH == 0;
  if (in.kind == IN_INT8 && in.lut_scale != 0.f)
    (tile ? launch_fwd_pair_t<N1, IN_INT8, true, true> : launch_fwd_pair_t<N1, IN_INT8, true, false>) (
        in, lut, nkeep, part0, nbatch, n2, tw4, scratch, apod, nsm, st);
  else if (in.kind == IN_INT8)
    (tile ? launch_fwd_pair_t<N1, IN_INT8, false, true> : launch_fwd_pair_t<N1, IN_INT8, false, false>) (
        in, lut, nkeep, part0, nbatch, n2, tw4, scratch, apod, nsm, st);
  else if (in.kind == IN_INT16)
    (tile ? launch_fwd_pair_t<N1, IN_INT16, false, true> : launch_fwd_pair_t<N1, IN_INT16, false, false>) (
        in, lut, nkeep, part0, nbatch, n2, tw4, scratch, apod, nsm, st);
  else
    launch_fwd_pair_t<N1, IN_FLOAT, false, false> (in, lut, nkeep, part0, nbatch, n2, tw4, scratch,
                                                   apod, nsm, st);
}

} // namespace

} // namespace b200
