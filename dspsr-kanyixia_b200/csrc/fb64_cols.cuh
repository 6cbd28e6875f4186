// fb64_cols.cuh -- forward column pass with the 64-channel filterbank in front
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"
#include "fwd_cols_pair.cuh"

namespace b200 {

namespace {

// K1 with the filterbank in front (Filterbank with freq_res 1 and 64 channels,
// FilterbankEngineCPU.C:379-535, then the first four-step pass of each
// channel's convolution), for raw TFPD input of one channel and two
// polarisations and n1 = 8 or 16.  The filterbank's own output never reaches
// memory: a warp takes one column i2 of one part and computes, for the eight
// filterbank samples t0 + j*n2 of that column, all 64 channels of both
// polarisations, then each channel's 8-point column DFT.
//
// Lane (j, q), j = lane/4, q = lane%4, reads raw samples s = q + 4m (m < 16)
// of filterbank sample j: a 16-point DFT over m (both polarisations packed)
// and the twiddle w64^(q ka) give Y[q][ka] (ka < 16).  One transpose through
// the warp's shared buffer hands lane 2 ka + pol the 32 values Y[q][ka] of
// every (q, j): 4-point DFTs over q give channels c = ka + 16 kb (kb < 4) of
// each filterbank sample, and 8-point DFTs over j the four channels' column
// DFTs, all in registers (64-point DFT as 16 x 4, X[ka + 16 kb] =
// sum_q w4^(q kb) w64^(q ka) Y[q][ka]).
//
// n1 = 16 splits each column's 16 samples by their first radix-2 step, which
// commutes with the filterbank: the block of half 0 transforms x_j + x_(j+8)
// and gives the even rows k1, the block of half 1 (x_j - x_(j+8)) w16^j and
// gives the odd ones.  Both read the raw samples (4 bytes each, the second
// time from L2) and do the work of an n1 = 8 column on them.
//
// The block's eight warps (eight consecutive columns) stage their outputs in
// shared memory and write each scratch row in runs of 64 bytes.  The
// transpose's rows are 34 float2 apart, so its stores (one row, 32 lanes) and
// 16-byte loads (32 rows) are free of bank conflicts.  The staging is
// column-major with the even and odd rows in two halves (row -> row/2 + (row
// odd) FBC_SODD, column stride FBC_SP odd): the 16 rows a half-warp stores and
// the 2 x 8 (row, column) pairs it loads for the write-out then fall in 16
// distinct bank pairs.  The pass is bound by the passes of its global and
// shared accesses through L1: with 4-byte raw loads (eight lines a warp each)
// and runs of 32 bytes (eight rows a warp) they were 640 per warp and column
// at n1 = 8, now 430: 922 us before, 895 us now for 134 M two-polarisation
// points at n1 = 8 and 985 us at n1 = 16 (the block's barriers are the largest
// stall).  An 8-bit table that is not affine is one 1 KB copy in shared memory
// (eight interleaved copies measured 10 % slower: the occupancy they cost
// outweighs the bank conflicts they remove).

constexpr int FBC_THREADS = 256;
constexpr int FBC_COLS = FBC_THREADS / 32;      // columns per block, one per warp
constexpr int FBC_XROW = 34;                    // exchange row stride (float2; 16-byte reads)
constexpr int FBC_XSTRIDE = 32 * FBC_XROW;      // float2 per warp exchange buffer
constexpr int FBC_SODD = 520;                   // staging offset of the odd rows (8 mod 16)
constexpr int FBC_SP = 1041;                    // staging column stride (odd)
constexpr size_t FBC_SMEM =
    (size_t (FBC_SP) * FBC_COLS > size_t (FBC_COLS) * FBC_XSTRIDE ? size_t (FBC_SP) * FBC_COLS
                                                                  : size_t (FBC_COLS) * FBC_XSTRIDE)
    * sizeof (float2);

__host__ __device__ constexpr int fbc_stage (int row, int col)
{
  return col * FBC_SP + (row >> 1) + (row & 1) * FBC_SODD;
}

// 4 x 4 transpose among the four lanes of a quad (q = lane % 4): lane q gets
// word q of each lane's four, in lane order
__device__ __forceinline__ void quad_transpose (uint4& w, unsigned q)
{
  const bool o1 = q & 1, o2 = q & 2;
  unsigned a = __shfl_xor_sync (FULL, o1 ? w.x : w.y, 1);
  unsigned b = __shfl_xor_sync (FULL, o1 ? w.z : w.w, 1);
  w = o1 ? make_uint4 (a, w.y, b, w.w) : make_uint4 (w.x, a, w.z, b);
  a = __shfl_xor_sync (FULL, o2 ? w.x : w.z, 2);
  b = __shfl_xor_sync (FULL, o2 ? w.y : w.w, 2);
  w = o2 ? make_uint4 (a, b, w.z, w.w) : make_uint4 (w.x, w.y, a, b);
}

// The 16 raw samples q + 4 m of one filterbank sample (r: its 64 samples).
// Where the sample starts on 16 bytes each lane loads four samples at a time
// and the quad transposes them.
template <int KIND>
__device__ __forceinline__ void load_raw16 (const typename RawPair<KIND>::T* r, unsigned q, bool wide,
                                            typename RawPair<KIND>::T* w)
{
  if constexpr (KIND == IN_INT8)
  {
    if (wide)
    {
#pragma unroll
      for (int i = 0; i < 4; i++)
      {
        uint4 x = __ldg (reinterpret_cast<const uint4*> (r) + 4 * i + q);
        quad_transpose (x, q);
        w[4 * i] = x.x;
        w[4 * i + 1] = x.y;
        w[4 * i + 2] = x.z;
        w[4 * i + 3] = x.w;
      }
      return;
    }
  }
#pragma unroll
  for (int m = 0; m < 16; m++) w[m] = __ldg (r + q + 4 * m);
}

template <int N1, int KIND, bool AFFINE>
__global__ void __launch_bounds__ (FBC_THREADS, 3)
k_fwd_cols_fb64 (const InputView in, const float* __restrict__ lut, const uint64_t nkeep,
                 const uint64_t part0, const unsigned n2, const float2* __restrict__ tw4,
                 float2* __restrict__ scratch)
{
  using Raw = typename RawPair<KIND>::T;
  extern __shared__ __align__ (16) float2 s_fbc[];
  __shared__ float s_lut[KIND == IN_INT8 && !AFFINE ? 256 : 1];
  __shared__ float2 s_tw64[64];
  if (KIND == IN_INT8 && !AFFINE)
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
      s_lut[i] = lut[i];
  if (threadIdx.x < 64)
    s_tw64[threadIdx.x] = make_float2 (cos64 (int (threadIdx.x)), -sin64 (int (threadIdx.x)));
  __syncthreads ();
  const UnpackPair u {s_lut, in.lut_scale, in.offset_binary ? 0u : 0x80008000u};
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned j = lane >> 2, q = lane & 3;
  constexpr unsigned HALVES = N1 / 8;
  const unsigned half = blockIdx.x % HALVES;
  const unsigned i0 = blockIdx.x / HALVES * FBC_COLS;
  const unsigned i2 = i0 + warp;
  const unsigned b = blockIdx.y;
  const uint64_t N = uint64_t (N1) * n2;
  float2* xb = s_fbc + warp * FBC_XSTRIDE;

  // the 64 raw samples of filterbank sample t lie in one segment of the input;
  // both segments start on 16 bytes (the carry always does) or the samples
  // are loaded one by one
  const bool wide = reinterpret_cast<uintptr_t> (in.main) % 16 == 0;
  const auto raw_of = [&] (uint64_t t) {
    return t < in.npre ? static_cast<const Raw*> (in.pre) + t * 64
                       : static_cast<const Raw*> (in.main) + (t - in.npre) * 64;
  };
  const uint64_t t = (part0 + b) * nkeep + i2 + uint64_t (j) * n2;
  C2 x[16];
  {
    Raw w0[16];
    load_raw16<KIND> (raw_of (t), q, wide, w0);
    if constexpr (N1 == 8)
    {
#pragma unroll
      for (int m = 0; m < 16; m++) x[m] = unpack_pair<KIND, AFFINE> (w0[m], u);
    }
    else
    {
      Raw w1[16];
      load_raw16<KIND> (raw_of (t + 8ull * n2), q, wide, w1);
      if (half == 0)
      {
#pragma unroll
        for (int m = 0; m < 16; m++)
          x[m] = dft::add (unpack_pair<KIND, AFFINE> (w0[m], u), unpack_pair<KIND, AFFINE> (w1[m], u));
      }
      else
      {
        const float2 w = s_tw64[4 * j];               // w16^j
#pragma unroll
        for (int m = 0; m < 16; m++)
          x[m] = dft::mulc (dft::sub (unpack_pair<KIND, AFFINE> (w0[m], u),
                                      unpack_pair<KIND, AFFINE> (w1[m], u)), w.x, w.y);
      }
    }
  }
  dft::run<16, -1> (x);
  // twiddle w64^(q ka); lane (j, q) then hands Y[q][ka] of both
  // polarisations to lane 2 ka + pol through the warp's buffer (row 2 ka + pol,
  // column 4 j + q, rows FBC_XROW float2 apart)
#pragma unroll
  for (int ka = 0; ka < 16; ka++)
  {
    const float2 w = s_tw64[(q * ka) & 63];
    const float2 a = make_float2 (x[ka].re.x, x[ka].im.x), c = make_float2 (x[ka].re.y, x[ka].im.y);
    xb[(2 * ka) * FBC_XROW + lane] = ka ? cmul (a, w) : a;
    xb[(2 * ka + 1) * FBC_XROW + lane] = ka ? cmul (c, w) : c;
  }
  __syncwarp ();
  // lane 2 ka + pol reads its row in 16-byte pairs: z[jj][qq] = Y[qq][ka] of
  // filterbank sample jj; 4-point DFTs over q: z[jj][kb] = channel ka + 16 kb
  // of filterbank sample jj
  float2 col[4][8];
#pragma unroll
  for (int jj = 0; jj < 8; jj++)
  {
    const float4 a = *reinterpret_cast<const float4*> (xb + lane * FBC_XROW + 4 * jj);
    const float4 c = *reinterpret_cast<const float4*> (xb + lane * FBC_XROW + 4 * jj + 2);
    float2 z[4] = {make_float2 (a.x, a.y), make_float2 (a.z, a.w), make_float2 (c.x, c.y),
                   make_float2 (c.z, c.w)};
    dft::run<4, -1> (z);
#pragma unroll
    for (int kb = 0; kb < 4; kb++) col[kb][jj] = z[kb];
  }
  // the column DFTs over the eight filterbank samples, per channel
#pragma unroll
  for (int kb = 0; kb < 4; kb++) dft::run<8, -1> (col[kb]);
  // four-step twiddle w_N^(k1 n2) of column i2 with the filterbank
  // normaliser 1/sqrt(64) (exact)
  float2 tw[8];
#pragma unroll
  for (int m = 0; m < 8; m++)
  {
    const unsigned k1 = HALVES * m + half;
    const float2 w = k1 ? __ldg (tw4 + uint64_t (k1) * n2 + i2) : make_float2 (1.f, 0.f);
    tw[m] = make_float2 (0.125f * w.x, 0.125f * w.y);
  }
  __syncthreads ();                    // every warp is done with its exchange buffer
  // channel c = ka + 16 kb, pol of lane 2 ka + pol; staging row
  // m*128 + c*2 + pol, column = warp
  {
    const unsigned ka = lane >> 1, pol = lane & 1;
#pragma unroll
    for (int kb = 0; kb < 4; kb++)
    {
      const unsigned c = ka + 16 * kb;
#pragma unroll
      for (int m = 0; m < 8; m++)
        s_fbc[fbc_stage (m * 128 + c * 2 + pol, warp)] = cmul (col[kb][m], tw[m]);
    }
  }
  __syncthreads ();
  // scratch row ((b*64 + c)*2 + pol)*N + k1*n2, columns i0 .. i0+FBC_COLS-1
#pragma unroll 4
  for (unsigned idx = threadIdx.x; idx < 1024 * FBC_COLS; idx += FBC_THREADS)
  {
    const unsigned row = idx / FBC_COLS, w = idx % FBC_COLS;
    const unsigned k1 = HALVES * (row >> 7) + half, c = (row & 127) >> 1, pol = row & 1;
    scratch[((uint64_t (b) * 64 + c) * 2 + pol) * N + uint64_t (k1) * n2 + i0 + w] =
        s_fbc[fbc_stage (row, w)];
  }
}

template <int N1, int KIND, bool AFFINE>
cudaError_t fb64_set_smem ()
{
  return cudaFuncSetAttribute (k_fwd_cols_fb64<N1, KIND, AFFINE>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, int (FBC_SMEM));
}

template <int N1>
cudaError_t fb64_setup_n1 ()
{
  cudaError_t e = fb64_set_smem<N1, IN_INT8, false> ();
  if (e == cudaSuccess) e = fb64_set_smem<N1, IN_INT8, true> ();
  if (e == cudaSuccess) e = fb64_set_smem<N1, IN_INT16, false> ();
  return e;
}

cudaError_t fb64_setup ()
{
  const cudaError_t e = fb64_setup_n1<8> ();
  return e == cudaSuccess ? fb64_setup_n1<16> () : e;
}

template <int N1>
void launch_fb64 (const InputView& in, const float* lut, uint64_t nkeep, uint64_t part0,
                  unsigned nbatch, unsigned n2, const float2* tw4, float2* scratch, cudaStream_t st)
{
  const dim3 g (n2 / FBC_COLS * (N1 / 8), nbatch);
  if (in.kind == IN_INT8 && in.lut_scale != 0.f)
    k_fwd_cols_fb64<N1, IN_INT8, true><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, lut, nkeep, part0, n2,
                                                                          tw4, scratch);
  else if (in.kind == IN_INT8)
    k_fwd_cols_fb64<N1, IN_INT8, false><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, lut, nkeep, part0,
                                                                           n2, tw4, scratch);
  else
    k_fwd_cols_fb64<N1, IN_INT16, false><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, lut, nkeep, part0,
                                                                            n2, tw4, scratch);
}

} // namespace

} // namespace b200
