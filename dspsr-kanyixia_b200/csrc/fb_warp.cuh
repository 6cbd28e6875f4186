// fb_warp.cuh -- FFT filterbank of 128 .. 1024 channels, 32 points per thread
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"

namespace b200 {

namespace {

// Filterbank with freq_res = 1 for NSUB = 32 M channels, M = 4 .. 32: M lanes
// of a warp transform one block of one polarisation with 32 points each,
// NSUB = 32 x M: lane t loads x[t + M r], a 32-point DFT over r, the twiddle
// w^(t q), one exchange through the warp's shared memory, then 32 / M M-point
// DFTs per lane give X[q + 32 p].  All of it meets at warp barriers only; the
// block's 8 * (32 / M) consecutive output samples of one polarisation are
// written together, so that every channel gets runs of 64 bytes and more.
// Persistent blocks keep the twiddle table.  Bound by HBM (8 or fewer bytes
// in, 8 out per value; TFPD samples of many channels by the 32-byte sector that
// each of them fetches from L2): 480 shared-memory clocks and 260 FP32 clocks per
// 1024 points against 730 of copying.  16 points per thread in three passes
// with block barriers took 1435 us for C5's block (134 M samples, 1024 channels,
// float), this 1033 us,
// and 951 us with the next tile's samples on their way to L2 meanwhile.
constexpr int FBW_WARPS = 8;

// bytes (a multiple of 16) from the 16-byte boundary at or before p
__device__ __forceinline__ void prefetch_l2_span (const void* p, unsigned bytes)
{
  const uint64_t a = reinterpret_cast<uint64_t> (p) & ~uint64_t (15);
  asm volatile ("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(bytes) : "memory");
}

template <int NSUB>
struct FbWarp
{
  static constexpr int M = NSUB / 32;
  static constexpr int G = 32 / M;                 // transforms per warp
  static constexpr int NB = FBW_WARPS * G;         // output samples per tile
  static constexpr int LD = M + 2;                 // exchange row stride: 16-byte reads of 8 rows
                                                   // fall in distinct banks at M = 32
  static constexpr int RS = 32 * LD + 2;           // region of one transform (2 mod 16)
  static constexpr size_t SMEM = (size_t (NB) * RS + NSUB) * sizeof (float2);
  static_assert (NB * RS % 2 == 0 && RS % 2 == 0, "16-byte aligned regions");
};

// TWO: both polarisations of TFPD samples in a tile, so that one load
// instruction takes them from the same sectors (a warp's first transforms are of
// one, the others of the other; the regions of one lie together)
template <int NSUB, int KIND, bool TWO>
__global__ void __launch_bounds__ (FBW_WARPS * 32, 2)
k_filterbank_warp (const InputView in, const float* __restrict__ lut, const uint64_t nblk,
                   const float scale, float2* __restrict__ out, const uint64_t out_span,
                   const uint64_t tiles_per_row, const uint64_t ntile)
{
  using F = FbWarp<NSUB>;
  constexpr int M = F::M;
  extern __shared__ __align__ (16) float2 s_fbw[];
  float2* tw = s_fbw + F::NB * F::RS;              // w_NSUB^(q t) at [q * M + t]
  __shared__ float s_lut[KIND == IN_INT8 ? 256 : 1];
  if constexpr (KIND == IN_INT8) load_lut (in, lut, s_lut);
  for (int i = threadIdx.x; i < NSUB; i += FBW_WARPS * 32)
  {
    double sn, cs;
    sincospi (-2.0 * double ((i / M) * (i % M)) / double (NSUB), &sn, &cs);
    tw[i] = make_float2 (float (cs), float (sn));
  }
  __syncthreads ();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned npol = in.npol;
  const uint64_t rowv = uint64_t (in.nchan) * npol;      // TFPD values per time sample
  static_assert (!TWO || (KIND != IN_FLOAT && F::G >= 2), "two transforms of a warp");
  constexpr int G = TWO ? F::G / 2 : F::G, NBT = FBW_WARPS * G;        // output samples: warp, tile
  const int t = lane % M, grp = lane / M;
  const int spol = TWO ? grp / G : 0, slot = warp * G + (TWO ? grp % G : grp);
  float2* s = s_fbw + (spol * NBT + slot) * F::RS;
  for (uint64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x)
  {
    // input channel and polarisation: outermost for FPT rows, innermost for TFPD
    // samples, whose sectors hold several rows: blocks at work together then
    // share them through L2 (32 dual-polarisation int8 channels into 512 each,
    // 64 M values: 768 us with the row outermost, 491 innermost, 352 with both
    // polarisations in a tile; into 128 each 1350, 668 and 483)
    const uint64_t nrow = TWO ? uint64_t (in.nchan) : rowv;
    const unsigned trow = unsigned (KIND == IN_FLOAT ? tile / tiles_per_row : tile % nrow);
    const uint64_t blk0 = (KIND == IN_FLOAT ? tile % tiles_per_row : tile / nrow) * NBT;
    const unsigned row = TWO ? 2 * trow + spol : trow;
    const bool live = blk0 + slot < nblk;
    const uint64_t t0 = (blk0 + slot) * NSUB + t;
    CP v[32];
#pragma unroll
    for (int r = 0; r < 32; r++)
    {
      float2 x = make_float2 (0.f, 0.f);
      if constexpr (KIND == IN_FLOAT)
      {
        if (live) x = __ldcs (static_cast<const float2*> (in.main) + row * in.main_span + t0 + M * r);
      }
      else
      {
        const uint64_t idx = (t0 + M * r) * rowv + row;
        if constexpr (KIND == IN_INT16)
        {
          const uint32_t w = live ? __ldg (static_cast<const uint32_t*> (in.main) + idx) : 0u;
          short re = short (w & 0xffff), im = short (w >> 16);
          if (in.offset_binary)
          {
            re = short (re ^ 0x8000);
            im = short (im ^ 0x8000);
          }
          // SixteenBitUnpacker.C:69: float(x) + 0.5
          x = make_float2 (__fadd_rn (float (re), 0.5f), __fadd_rn (float (im), 0.5f));
        }
        else
        {
          const unsigned w = live ? __ldg (static_cast<const unsigned short*> (in.main) + idx) : 0u;
          x = make_float2 (s_lut[w & 0xff], s_lut[w >> 8]);
        }
      }
      v[r].z = x;
    }
    if constexpr (KIND == IN_FLOAT)
    {
      // the transform this lane's slot takes next starts on its way to L2
      const uint64_t nt = tile + gridDim.x;
      const uint64_t nb0 = nt % tiles_per_row * NBT + slot;
      if (t == 0 && nt < ntile && nb0 < nblk)
        prefetch_l2_span (static_cast<const float2*> (in.main)
                              + nt / tiles_per_row * in.main_span + nb0 * NSUB, NSUB * 8);
    }
    dft::run<32, -1> (v);
#pragma unroll
    for (int q = 0; q < 32; q++) s[q * F::LD + t] = q ? cmul (v[q].z, tw[q * M + t]) : v[q].z;
    __syncwarp ();
    // rows q = t + M i of the exchange, M values each
#pragma unroll
    for (int i = 0; i < F::G; i++)
#pragma unroll
      for (int j = 0; j < M / 2; j++)
      {
        const float4 x = *reinterpret_cast<const float4*> (s + (t + M * i) * F::LD + 2 * j);
        v[i * M + 2 * j].z = make_float2 (x.x, x.y);
        v[i * M + 2 * j + 1].z = make_float2 (x.z, x.w);
      }
    __syncwarp ();
#pragma unroll
    for (int i = 0; i < F::G; i++)
    {
      dft::run<M, -1> (v + i * M);
#pragma unroll
      for (int p = 0; p < M; p++) s[t + M * i + 32 * p] = v[i * M + p].z;
    }
    __syncthreads ();
    const unsigned nb = unsigned (min (uint64_t (NBT), nblk - blk0));
    const unsigned cin = TWO ? trow : row / npol, p0 = TWO ? 0 : row % npol;
    float2* o = out + (uint64_t (cin) * NSUB * npol + p0) * out_span + blk0;
#pragma unroll 8
    for (unsigned e = threadIdx.x; e < unsigned (F::NB * NSUB); e += FBW_WARPS * 32)
    {
      const unsigned b = e % unsigned (NBT), k = e / unsigned (TWO ? F::NB : NBT);
      const unsigned p = TWO ? e / unsigned (NBT) % 2 : 0;
      const float2 y = s_fbw[(TWO ? p * NBT + b : b) * F::RS + k];
      if (b < nb)
        o[(TWO ? uint64_t (k) * 2 + p : uint64_t (k) * npol) * out_span + b] =
            make_float2 (__fmul_rn (scale, y.x), __fmul_rn (scale, y.y));
    }
    __syncthreads ();                  // the regions are free again
  }
}

} // namespace

} // namespace b200
