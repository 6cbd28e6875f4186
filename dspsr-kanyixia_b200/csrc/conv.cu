// conv.cu -- overlap-save convolution kernels of the B200 baseband hot path.
//
// Overlap-save coherent dedispersion (Signal/General/Convolution.C:724-803 is
// the CPU algorithm; CUDA::ConvolutionEngine runs it as cuFFT + 3 kernels per
// batch) is restructured here as a four-step FFT of length N = n1 * n2:
//
//   K1 (columns)  unpack the int8/int16/float input on load, n1-point DFTs in
//                 registers across the n1 chunks of n2 samples, store rows k1.
//   K2 (rows)     twiddle w_N^{k1 n2}, n2-point Stockham FFT in shared memory,
//                 multiply by the response (stored in four-step order), inverse
//                 n2-point FFT, conjugate twiddle -- one read and one write.
//   K3 (columns)  inverse n1-point DFTs in registers, overlap discard, and then
//                 either write the voltages (Engine::perform) or detect and
//                 fold in the same pass (warp-segmented reduction by bin).
//
// For n1 == 1 a single kernel does load, FFT, multiply, inverse FFT and the
// epilogue entirely in shared memory: one HBM round trip per part.
//
// FFT sign conventions are FFTW's (forward -1, backward +1, unnormalised); the
// 1/sqrt(N) normaliser is folded into the response, as Convolution::prepare
// does (Convolution.C:401-414).

#include "fwd_cols.cuh"
#include "fwd_cols_pair.cuh"
#include "inv_cols_split.cuh"
#include "rows32.cuh"

namespace b200 {

namespace {

// --------------------------------------------------------------------------
// shared-memory Stockham FFT
// --------------------------------------------------------------------------

template <int N, int T, int D, int P>
__device__ __forceinline__ void smem_pass (float2* s, float2* v, const float2* tw)
{
  if constexpr (P < stockham_npass (N))
  {
    constexpr int R = stockham_radix (N, P);
    constexpr int Ns = stockham_ns (N, P);
    StockhamPass<N, R, T, D>::load (threadIdx.x, s, v);
    __syncthreads ();
    StockhamPass<N, R, T, D>::compute_store (threadIdx.x, Ns, v, s, tw);
    __syncthreads ();
    smem_pass<N, T, D, P + 1> (s, v, tw);
  }
}

// N-point FFT of s[spad(0..N-1)] in place; the caller has synchronised after
// writing s.  Returns synchronised.
template <int N, int T, int D>
__device__ __forceinline__ void smem_fft (float2* s, const float2* tw)
{
  float2 v[N / T];
  smem_pass<N, T, D, 0> (s, v, tw);
}

// --------------------------------------------------------------------------
// K1 with the filterbank in front (Filterbank with freq_res 1 and 64 channels,
// FilterbankEngineCPU.C:379-535, then the first four-step pass of each
// channel's convolution), for raw TFPD input of one channel and two
// polarisations and n1 = 8.  The filterbank's own output never reaches
// memory: a warp takes one column i2 of one part and computes, for the eight
// filterbank samples t0 + j*n2 of that column, all 64 channels of both
// polarisations, then each channel's 8-point column DFT.
//
// Lane (j, q), j = lane/4, q = lane%4, reads raw samples s = q + 4m (m < 16)
// of filterbank sample j: a 16-point DFT over m and the twiddle w64^(q ka)
// give Y[q][ka] (ka < 16).  One transpose through the warp's shared buffer
// hands lane 2 ka + pol the 32 values Y[q][ka] of every (q, j): 4-point DFTs
// over q give channels c = ka + 16 kb (kb < 4) of each filterbank sample,
// and 8-point DFTs over j the four channels' column DFTs, all in registers
// (64-point DFT as 16 x 4, X[ka + 16 kb] = sum_q w4^(q kb) w64^(q ka)
// Y[q][ka]).  The block's four warps (four consecutive
// columns) stage their outputs in shared memory and write each scratch row
// in runs of one 32-byte sector (blocks of two or eight warps measured
// slower).  The transpose's rows are 34 float2 apart, so its stores (one row,
// 32 lanes) and 16-byte loads (32 rows) are free of bank conflicts.  The staging is column-major with the even and odd rows in two
// halves (row -> row/2 + (row odd) FBC_SODD, column stride FBC_SP = 2 mod 16):
// the 16 rows a half-warp stores (two apart) and the 4 x 4 (row, column)
// pairs it loads for the write-out then fall in 16 distinct bank pairs.
// --------------------------------------------------------------------------

constexpr int FBC_THREADS = 128;
constexpr int FBC_COLS = FBC_THREADS / 32;      // columns per block, one per warp
constexpr int FBC_XROW = 34;                    // exchange row stride (float2; 16-byte reads)
constexpr int FBC_XSTRIDE = 32 * FBC_XROW;      // float2 per warp exchange buffer
constexpr int FBC_SODD = 520;                   // staging offset of the odd rows (8 mod 16)
constexpr int FBC_SP = 1042;                    // staging column stride (2 mod 16)
constexpr size_t FBC_SMEM =
    (size_t (FBC_SP) * FBC_COLS > size_t (FBC_COLS) * FBC_XSTRIDE ? size_t (FBC_SP) * FBC_COLS
                                                                  : size_t (FBC_COLS) * FBC_XSTRIDE)
    * sizeof (float2);

__host__ __device__ constexpr int fbc_stage (int row, int col)
{
  return col * FBC_SP + (row >> 1) + (row & 1) * FBC_SODD;
}

// (float(x) + 0.5f) * scale for the two's-complement byte x, bit for bit:
// 2^22 + (x + 128) has its last mantissa bit worth 0.5, so subtracting
// 2^22 + 127.5 leaves x + 0.5 exactly; no int -> float conversion
__device__ __forceinline__ float unpack_affine (unsigned byte, float scale)
{
  const float big = __int_as_float (0x4a800000u | (((byte & 0xffu) ^ 0x80u) << 1));
  return __fmul_rn (__fsub_rn (big, 4194431.5f), scale);
}

// The 8-bit table of the fused filterbank pass is one 1 KB copy in shared
// memory.  Eight interleaved copies (lane l reading copy l % 8, so a warp's
// random lookups spread over all banks) measured 10 % slower on the C2 pass:
// the 8 KB table costs more in occupancy than the bank conflicts it removes.

template <int KIND, bool AFFINE>
__device__ __forceinline__ void fetch_raw2 (const InputView& in, const float* s_lut, uint64_t r,
                                            float2& p0, float2& p1)
{
  const void* base = in.main;
  const uint64_t npre = in.npre * 64;
  if (r < npre)
    base = in.pre;
  else
    r -= npre;
  if constexpr (KIND == IN_INT8)
  {
    const unsigned w = __ldg (static_cast<const unsigned*> (base) + r);
    if constexpr (AFFINE)
    {
      const float sc = in.lut_scale;
      p0 = make_float2 (unpack_affine (w, sc), unpack_affine (w >> 8, sc));
      p1 = make_float2 (unpack_affine (w >> 16, sc), unpack_affine (w >> 24, sc));
    }
    else
    {
      p0 = make_float2 (s_lut[w & 0xff], s_lut[(w >> 8) & 0xff]);
      p1 = make_float2 (s_lut[(w >> 16) & 0xff], s_lut[w >> 24]);
    }
  }
  else
  {
    const uint2 w = __ldg (static_cast<const uint2*> (base) + r);
    short a = short (w.x & 0xffff), b = short (w.x >> 16);
    short c = short (w.y & 0xffff), d = short (w.y >> 16);
    if (in.offset_binary)
    {
      a = short (a ^ 0x8000);
      b = short (b ^ 0x8000);
      c = short (c ^ 0x8000);
      d = short (d ^ 0x8000);
    }
    p0 = make_float2 (__fadd_rn (float (a), 0.5f), __fadd_rn (float (b), 0.5f));
    p1 = make_float2 (__fadd_rn (float (c), 0.5f), __fadd_rn (float (d), 0.5f));
  }
}

template <int KIND, bool AFFINE>
__global__ void __launch_bounds__ (FBC_THREADS, 768 / FBC_THREADS)
k_fwd_cols_fb64 (const InputView in, const float* __restrict__ lut, const uint64_t nkeep,
                 const uint64_t part0, const unsigned n2, const float2* __restrict__ tw4,
                 float2* __restrict__ scratch)
{
  extern __shared__ __align__ (16) float2 s_fbc[];
  __shared__ float s_lut[AFFINE ? 1 : 256];
  __shared__ float2 s_tw64[64];
  if (!AFFINE && in.kind == IN_INT8)
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
      s_lut[i] = lut[i];
  if (threadIdx.x < 64)
    s_tw64[threadIdx.x] = make_float2 (cos64 (int (threadIdx.x)), -sin64 (int (threadIdx.x)));
  __syncthreads ();
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned j = lane >> 2, q = lane & 3;
  const unsigned i0 = blockIdx.x * FBC_COLS;
  const unsigned i2 = i0 + warp;
  const unsigned b = blockIdx.y;
  const uint64_t N = 8ull * n2;
  float2* xb = s_fbc + warp * FBC_XSTRIDE;

  // raw samples q + 4m of filterbank sample t, both polarisations
  const uint64_t t = (part0 + b) * nkeep + i2 + uint64_t (j) * n2;
  float2 x0[16], x1[16];
#pragma unroll
  for (int m = 0; m < 16; m++)
    fetch_raw2<KIND, AFFINE> (in, s_lut, t * 64 + q + 4 * m, x0[m], x1[m]);
  RegDFT<16, -1>::run (x0);
  RegDFT<16, -1>::run (x1);
  // twiddle w64^(q ka); lane (j, q) then hands Y[q][ka] of both
  // polarisations to lane 2 ka + pol through the warp's buffer (row 2 ka + pol,
  // column 4 j + q, rows FBC_XROW float2 apart)
#pragma unroll
  for (int ka = 0; ka < 16; ka++)
  {
    const float2 w = s_tw64[(q * ka) & 63];
    xb[(2 * ka) * FBC_XROW + lane] = cmul (x0[ka], w);
    xb[(2 * ka + 1) * FBC_XROW + lane] = cmul (x1[ka], w);
  }
  __syncwarp ();
  // lane 2 ka + pol reads its row in 16-byte pairs: z[jj][qq] = Y[qq][ka] of
  // filterbank sample jj
  float2 z[8][4];
#pragma unroll
  for (int jj = 0; jj < 8; jj++)
#pragma unroll
    for (int qq = 0; qq < 4; qq += 2)
    {
      const float4 t = *reinterpret_cast<const float4*> (xb + lane * FBC_XROW + 4 * jj + qq);
      z[jj][qq] = make_float2 (t.x, t.y);
      z[jj][qq + 1] = make_float2 (t.z, t.w);
    }
  // 4-point DFTs over q: z[jj][kb] = channel ka + 16 kb of filterbank sample jj
#pragma unroll
  for (int jj = 0; jj < 8; jj++) RegDFT<4, -1>::run (z[jj]);
  // the column DFTs over the eight filterbank samples, per channel
  float2 col[4][8];
#pragma unroll
  for (int kb = 0; kb < 4; kb++)
  {
#pragma unroll
    for (int jj = 0; jj < 8; jj++) col[kb][jj] = z[jj][kb];
    RegDFT<8, -1>::run (col[kb]);
  }
  // four-step twiddle w_N^(k1 n2) of column i2, and the filterbank
  // normaliser 1/sqrt(64) (exact)
  float2 tw[8];
  tw[0] = make_float2 (1.f, 0.f);
#pragma unroll
  for (int k1 = 1; k1 < 8; k1++) tw[k1] = __ldg (tw4 + uint64_t (k1) * n2 + i2);
  __syncthreads ();                    // every warp is done with its exchange buffer
  // channel c = ka + 16 kb, pol of lane 2 ka + pol; staging row
  // k1*128 + c*2 + pol, column = warp
  {
    const unsigned ka = lane >> 1, pol = lane & 1;
#pragma unroll
    for (int kb = 0; kb < 4; kb++)
    {
      const unsigned c = ka + 16 * kb;
#pragma unroll
      for (int k1 = 0; k1 < 8; k1++)
      {
        float2 o = k1 ? cmul (col[kb][k1], tw[k1]) : col[kb][k1];
        o = make_float2 (__fmul_rn (o.x, 0.125f), __fmul_rn (o.y, 0.125f));
        s_fbc[fbc_stage (k1 * 128 + c * 2 + pol, warp)] = o;
      }
    }
  }
  __syncthreads ();
  // scratch row ((b*64 + c)*2 + pol)*N + k1*n2, columns i0 .. i0+FBC_COLS-1
#pragma unroll 4
  for (unsigned idx = threadIdx.x; idx < 1024 * FBC_COLS; idx += FBC_THREADS)
  {
    const unsigned row = idx / FBC_COLS, w = idx % FBC_COLS;
    const unsigned k1 = row >> 7, c = (row & 127) >> 1, pol = row & 1;
    scratch[((uint64_t (b) * 64 + c) * 2 + pol) * N + uint64_t (k1) * n2 + i0 + w] =
        s_fbc[fbc_stage (row, w)];
  }
}

// --------------------------------------------------------------------------
// K3: inverse column DFTs, overlap discard, voltage out or detect + fold
// --------------------------------------------------------------------------

template <int N1, int NPOL, int MODE, int NOUT>
__global__ void __launch_bounds__ (128, N1 >= 32 ? 3 : 4)
k_inv_cols (const float2* __restrict__ scratch, const unsigned n2, const unsigned nchan,
            const uint64_t nkeep, const unsigned nfilt_pos, const uint64_t part0,
            const float2* __restrict__ tw4, const FoldView fv, const VoltView vv)
{
  const unsigned b = blockIdx.y;
  const unsigned c = blockIdx.z;
  const uint64_t N = uint64_t (N1) * n2;
  const uint64_t tbase0 = (part0 + b) * nkeep;
  float* prof = fv.profiles + uint64_t (c) * NOUT * fv.stride;
  unsigned* hits = c == 0 ? fv.hits : nullptr;
  if constexpr (N1 == 32)
  {
    // Two threads per column (16 columns per warp): thread h = lane & 1 of a
    // pair takes rows 2m + h, a 16-point inverse DFT of them gives E (h = 0)
    // or O (h = 1), thread 1 applies w32^j, one exchange leaves
    // X[j] = E[j] + w32^j O[j] with thread 0 and X[j + 16] = E[j] - w32^j O[j]
    // with thread 1; a second shuffle moves them so that lanes 0..15 hold
    // X[j] of the warp's 16 columns and lanes 16..31 X[j + 16] (runs of
    // consecutive samples for the fold).
    const unsigned lane = threadIdx.x & 31;
    const unsigned h = lane & 1;
    const unsigned colw = blockIdx.x * 64 + (threadIdx.x >> 5) * 16;
    const unsigned i2 = colw + (lane >> 1);
    float2 v[NPOL][16];
#pragma unroll
    for (int m = 0; m < 16; m++)
    {
      const unsigned k = 2 * m + h;
      const float2 w = __ldg (tw4 + uint64_t (k) * n2 + i2);
#pragma unroll
      for (int p = 0; p < NPOL; p++)
      {
        const float2 x = scratch[((uint64_t (b) * nchan + c) * NPOL + p) * N + uint64_t (k) * n2 + i2];
        v[p][m] = k ? cmulc (x, w) : x;
      }
    }
    const int srcl = lane < 16 ? 2 * int (lane) : 2 * (int (lane) - 16) + 1;
#pragma unroll
    for (int p = 0; p < NPOL; p++)
    {
      RegDFT<16, +1>::run (v[p]);
#pragma unroll
      for (int j = 0; j < 16; j++)
      {
        const float2 mine = h ? tw_mul<32, +1> (j, v[p][j]) : v[p][j];
        const float2 other = make_float2 (__shfl_xor_sync (FULL, mine.x, 1),
                                          __shfl_xor_sync (FULL, mine.y, 1));
        const float2 x = h ? csub (other, mine) : cadd (mine, other);
        v[p][j] = make_float2 (__shfl_sync (FULL, x.x, srcl), __shfl_sync (FULL, x.y, srcl));
      }
    }
    const unsigned ocol = colw + (lane & 15), koff = 16 * (lane >> 4);
#pragma unroll
    for (int j = 0; j < 16; j++)
    {
      const uint64_t tl = uint64_t (koff + j) * n2 + ocol;
      const bool ok = tl >= nfilt_pos && tl < nfilt_pos + nkeep;
      const uint64_t t = tbase0 + (tl - nfilt_pos);
      if constexpr (MODE == OUT_VOLTAGE)
      {
        if (ok)
        {
#pragma unroll
          for (int p = 0; p < NPOL; p++)
            vv.out[(uint64_t (c) * NPOL + p) * vv.span + t] = v[p][j];
        }
      }
      else
        detect_fold<NOUT> (fv, NPOL, fold_column (fv, ok, t), v[0][j], v[NPOL - 1][j], prof, hits);
    }
    return;
  }
  const unsigned i2 = blockIdx.x * blockDim.x + threadIdx.x;
  float2 w[N1];
#pragma unroll
  for (int k = 1; k < N1; k++)
    w[k] = __ldg (tw4 + uint64_t (k) * n2 + i2);
  // the profile columns, asked for with the values
  unsigned fcol[MODE == OUT_FOLD ? N1 : 1];
  if constexpr (MODE == OUT_FOLD)
  {
#pragma unroll
    for (int k = 0; k < N1; k++)
    {
      const uint64_t tl = uint64_t (k) * n2 + i2;
      const bool ok = tl >= nfilt_pos && tl < nfilt_pos + nkeep;
      fcol[k] = fold_column (fv, ok, tbase0 + (tl - nfilt_pos));
    }
  }
  float2 v[NPOL][N1];
#pragma unroll
  for (int p = 0; p < NPOL; p++)
  {
    const float2* src = scratch + ((uint64_t (b) * nchan + c) * NPOL + p) * N + i2;
#pragma unroll
    for (int k = 0; k < N1; k++)
      v[p][k] = src[uint64_t (k) * n2];
  }
#pragma unroll
  for (int p = 0; p < NPOL; p++)
  {
    // conjugate four-step twiddle, then the inverse n1-point DFT
#pragma unroll
    for (int k = 1; k < N1; k++)
      v[p][k] = cmulc (v[p][k], w[k]);
    RegDFT<N1, +1>::run (v[p]);
  }
  const uint64_t tbase = (part0 + b) * nkeep;
#pragma unroll
  for (int k = 0; k < N1; k++)
  {
    const uint64_t tl = uint64_t (k) * n2 + i2;
    const bool ok = tl >= nfilt_pos && tl < nfilt_pos + nkeep;
    const uint64_t t = tbase + (tl - nfilt_pos);
    if constexpr (MODE == OUT_VOLTAGE)
    {
      if (ok)
      {
#pragma unroll
        for (int p = 0; p < NPOL; p++)
          vv.out[(uint64_t (c) * NPOL + p) * vv.span + t] = v[p][k];
      }
    }
    else
      detect_fold<NOUT> (fv, NPOL, fcol[k], v[0][k], v[NPOL - 1][k], prof, hits);
  }
}

// --------------------------------------------------------------------------
// single-kernel path (n1 == 1): everything in shared memory
// --------------------------------------------------------------------------

template <int N, int T, int KIND, int MODE, int NOUT>
__global__ void __launch_bounds__ (T, 512 / T)
k_fused (const InputView in, const float* __restrict__ lut, const float2* __restrict__ tw,
         const float2* __restrict__ H, const uint64_t nkeep, const unsigned nfilt_pos,
         const uint64_t part0, const FoldView fv, const VoltView vv,
         const float* __restrict__ apod)
{
  extern __shared__ float2 s[];
  __shared__ float s_lut[256];
  constexpr int SP = spad_size (N);
  const unsigned b = blockIdx.x;
  const unsigned c = blockIdx.y;
  const uint64_t part = part0 + b;
  const unsigned npol = in.npol;
  load_lut (in, lut, s_lut);
  __syncthreads ();
  for (unsigned p = 0; p < npol; p++)
    for (int i = threadIdx.x; i < N; i += T)
    {
      float2 x = fetch<KIND> (in, s_lut, c, p, part * nkeep + i);
      if (apod)
      {
        const float w = __ldg (apod + i);
        x = make_float2 (__fmul_rn (x.x, w), __fmul_rn (x.y, w));
      }
      s[p * SP + spad (i)] = x;
    }
  __syncthreads ();
  const float2* h = H + uint64_t (c) * N;
  for (unsigned p = 0; p < npol; p++)
  {
    float2* sp = s + p * SP;
    smem_fft<N, T, -1> (sp, tw);
    for (int i = threadIdx.x; i < N; i += T)
    {
      const float2 d = sp[spad (i)];
      const float2 f = __ldg (h + i);
      sp[spad (i)] = make_float2 (d.x * f.x - d.y * f.y, d.x * f.y + d.y * f.x);
    }
    __syncthreads ();
    smem_fft<N, T, +1> (sp, tw);
  }
  const uint64_t tbase = part * nkeep;
  float* prof = fv.profiles + uint64_t (c) * NOUT * fv.stride;
  unsigned* hits = c == 0 ? fv.hits : nullptr;
  const unsigned rounds = unsigned ((nkeep + T - 1) / T);
  for (unsigned r = 0; r < rounds; r++)
  {
    const uint64_t j = uint64_t (r) * T + threadIdx.x;
    const bool ok = j < nkeep;
    const int tl = ok ? int (nfilt_pos + j) : 0;
    const float2 pv = s[spad (tl)];
    const float2 qv = npol > 1 ? s[SP + spad (tl)] : make_float2 (0.f, 0.f);
    if (MODE == OUT_VOLTAGE)
    {
      if (ok)
      {
        vv.out[(uint64_t (c) * npol) * vv.span + tbase + j] = pv;
        if (npol > 1) vv.out[(uint64_t (c) * npol + 1) * vv.span + tbase + j] = qv;
      }
    }
    else
      detect_fold<NOUT> (fv, npol, fold_column (fv, ok, tbase + j), pv, qv, prof, hits);
  }
}

// --------------------------------------------------------------------------
// launch helpers
// --------------------------------------------------------------------------

template <int N1, int NPOL, int MODE, int NOUT>
void launch_inv (const ConvShape& sh, dim3 grid, float2* scratch, uint64_t part0,
                 const ConvTables& tb, const FoldView& fv, const VoltView& vv, cudaStream_t st)
{
  if constexpr (N1 >= 8 && NPOL == 2)
  {
    launch_inv_split<N1, MODE, NOUT> (scratch, {sh.n2, sh.n2, sh.nchan, sh.nkeep, sh.nfilt_pos},
                                      part0, grid.y, tb.tw4, tb.nsm, fv, vv, st);
    return;
  }
  else
  {
  if (N1 == 32) grid.x = sh.n2 / 64;        // two threads per column
  k_inv_cols<N1, NPOL, MODE, NOUT><<<grid, 128, 0, st>>> (scratch, sh.n2, sh.nchan, sh.nkeep,
                                                          sh.nfilt_pos, part0, tb.tw4, fv, vv);
  }
}

template <int N2>
void launch_rows (unsigned nrows, float2* scratch, const ConvTables& tb, unsigned n1,
                  const ConvShape& sh, cudaStream_t st)
{
  if (N2 == 8192 && tb.tc_splits)
  {
    launch_rows_mma (nrows, scratch, tb, n1, sh, st);
    return;
  }
  // persistent: as many CTAs as are resident at once
  const unsigned grid = std::min<unsigned> (nrows, rows_ctas_per_sm (N2) * unsigned (tb.nsm));
  k_rows32<N2, true><<<grid, Row32<N2>::T, rows32_smem_bytes<N2> (), st>>> (
      scratch, tb.H, n1, sh.nchan, sh.npol, nrows, nrows / (n1 * sh.nchan));
}

template <int N1>
cudaError_t run_fourstep_n1 (const ConvShape& sh, const ConvTables& tb, const InputView& in,
                             uint64_t part0, unsigned nbatch, float2* scratch, int mode,
                             const FoldView& fv, const VoltView& vv, cudaStream_t st,
                             const KernelClock* clk)
{
  const dim3 gcol (sh.n2 / 128, nbatch, sh.nchan);
  const dim3 gfwd (sh.n2 / fwd_cols_per_block<N1> (), nbatch, sh.nchan);
  if (in.fb_nsub)
  {
    // the 64-channel filterbank inside the column pass
    if (N1 != 8 || in.fb_nsub != 64 || sh.nchan != 64 || in.nchan != 1 || in.npol != 2
        || sh.npol != 2 || tb.apod || (in.kind != IN_INT8 && in.kind != IN_INT16))
      return cudaErrorInvalidValue;
    ClockScope cs (clk, KK_FWD_COLS, st);
    const dim3 g (sh.n2 / FBC_COLS, nbatch);
    if (in.kind == IN_INT8 && in.lut_scale != 0.f)
      k_fwd_cols_fb64<IN_INT8, true><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, tb.lut, sh.nkeep, part0,
                                                                         sh.n2, tb.tw4, scratch);
    else if (in.kind == IN_INT8)
      k_fwd_cols_fb64<IN_INT8, false><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, tb.lut, sh.nkeep, part0,
                                                                          sh.n2, tb.tw4, scratch);
    else
      k_fwd_cols_fb64<IN_INT16, false><<<g, FBC_THREADS, FBC_SMEM, st>>> (in, tb.lut, sh.nkeep,
                                                                           part0, sh.n2, tb.tw4,
                                                                           scratch);
  }
  else if (in.npol == 2 && fwd_pair_aligned (in))
  {
    ClockScope cs (clk, KK_FWD_COLS, st);
    launch_fwd_pair<N1> (in, tb.lut, sh.nkeep, part0, nbatch, sh.n2, tb.tw4, scratch, tb.apod,
                         tb.nsm, st);
  }
  else
  {
  ClockScope cs (clk, KK_FWD_COLS, st);
  if (in.kind == IN_INT8)
    k_fwd_cols<N1, IN_INT8><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.nkeep, part0, sh.n2, tb.tw4,
                                                   scratch, tb.apod);
  else if (in.kind == IN_INT16)
    k_fwd_cols<N1, IN_INT16><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.nkeep, part0, sh.n2, tb.tw4,
                                                    scratch, tb.apod);
  else
    k_fwd_cols<N1, IN_FLOAT><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.nkeep, part0, sh.n2, tb.tw4,
                                                    scratch, tb.apod);
  }
  const unsigned nrows = N1 * nbatch * sh.nchan * sh.npol;
  {
  ClockScope cs (clk, KK_ROWS, st);
  if (sh.n2 == 8192)
    launch_rows<8192> (nrows, scratch, tb, N1, sh, st);
  else if (sh.n2 == 4096)
    launch_rows<4096> (nrows, scratch, tb, N1, sh, st);
  else
    return cudaErrorInvalidValue;
  }
  ClockScope cs (clk, KK_INV_COLS, st);
  if (sh.npol == 2)
  {
    if (mode == OUT_VOLTAGE)
      launch_inv<N1, 2, OUT_VOLTAGE, 1> (sh, gcol, scratch, part0, tb, fv, vv, st);
    else if (fv.nout == 1)
      launch_inv<N1, 2, OUT_FOLD, 1> (sh, gcol, scratch, part0, tb, fv, vv, st);
    else if (fv.nout == 2)
      launch_inv<N1, 2, OUT_FOLD, 2> (sh, gcol, scratch, part0, tb, fv, vv, st);
    else
      launch_inv<N1, 2, OUT_FOLD, 4> (sh, gcol, scratch, part0, tb, fv, vv, st);
  }
  else
  {
    if (mode == OUT_VOLTAGE)
      launch_inv<N1, 1, OUT_VOLTAGE, 1> (sh, gcol, scratch, part0, tb, fv, vv, st);
    else
      launch_inv<N1, 1, OUT_FOLD, 1> (sh, gcol, scratch, part0, tb, fv, vv, st);
  }
  return cudaGetLastError ();
}

// The fused kernel's shared-memory opt-in (sized for two polarisations), once
// per device and instantiation; later calls only test a bit, so that calls
// made inside a stream capture set nothing up.
template <int N, int KIND, int MODE, int NOUT>
cudaError_t fused_setup ()
{
  static std::atomic<unsigned> done {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess) return e;
  const unsigned bit = dev < 32 ? 1u << dev : 0u;    // devices past 32: set every time
  if (bit && (done.load () & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute (k_fused<N, stockham_threads (N), KIND, MODE, NOUT>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                            int (2 * spad_size (N) * sizeof (float2)));
  if (e == cudaSuccess) done.fetch_or (bit);
  return e;
}

template <int N, int KIND, int MODE, int NOUT>
cudaError_t run_fused_t (const ConvShape& sh, const ConvTables& tb, const InputView& in,
                         uint64_t part0, unsigned nbatch, const FoldView& fv,
                         const VoltView& vv, cudaStream_t st, const KernelClock* clk)
{
  constexpr int T = stockham_threads (N);
  const size_t smem = size_t (in.npol) * spad_size (N) * sizeof (float2);
  auto kern = k_fused<N, T, KIND, MODE, NOUT>;
  cudaError_t err = fused_setup<N, KIND, MODE, NOUT> ();
  if (err != cudaSuccess) return err;
  ClockScope cs (clk, KK_FUSED, st);
  kern<<<dim3 (nbatch, sh.nchan), T, smem, st>>> (in, tb.lut, tb.tw2, tb.H, sh.nkeep,
                                                  sh.nfilt_pos, part0, fv, vv, tb.apod);
  return cudaGetLastError ();
}

template <int N, int KIND>
cudaError_t run_fused_k (const ConvShape& sh, const ConvTables& tb, const InputView& in,
                         uint64_t part0, unsigned nbatch, int mode, const FoldView& fv,
                         const VoltView& vv, cudaStream_t st, const KernelClock* clk)
{
  if (mode == OUT_VOLTAGE)
    return run_fused_t<N, KIND, OUT_VOLTAGE, 1> (sh, tb, in, part0, nbatch, fv, vv, st, clk);
  if (fv.nout == 1)
    return run_fused_t<N, KIND, OUT_FOLD, 1> (sh, tb, in, part0, nbatch, fv, vv, st, clk);
  if (fv.nout == 2)
    return run_fused_t<N, KIND, OUT_FOLD, 2> (sh, tb, in, part0, nbatch, fv, vv, st, clk);
  return run_fused_t<N, KIND, OUT_FOLD, 4> (sh, tb, in, part0, nbatch, fv, vv, st, clk);
}

template <int N>
cudaError_t run_fused (const ConvShape& sh, const ConvTables& tb, const InputView& in,
                       uint64_t part0, unsigned nbatch, int mode, const FoldView& fv,
                       const VoltView& vv, cudaStream_t st, const KernelClock* clk)
{
  if (in.kind == IN_INT8)
    return run_fused_k<N, IN_INT8> (sh, tb, in, part0, nbatch, mode, fv, vv, st, clk);
  if (in.kind == IN_INT16)
    return run_fused_k<N, IN_INT16> (sh, tb, in, part0, nbatch, mode, fv, vv, st, clk);
  return run_fused_k<N, IN_FLOAT> (sh, tb, in, part0, nbatch, mode, fv, vv, st, clk);
}

} // namespace

unsigned rows_ctas_per_sm (unsigned n2)
{
  return n2 == 8192 ? rows32_ctas_per_sm<8192> () : rows32_ctas_per_sm<4096> ();
}

// The four-step kernels' shared-memory opt-in, once per device (the current
// one); later calls only test a bit.
cudaError_t convolution_kernel_setup ()
{
  static std::atomic<unsigned> attr_done {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess) return e;
  const unsigned bit = dev < 32 ? 1u << dev : 0u;    // devices past 32: set every time
  if (bit && (attr_done.load () & bit)) return cudaSuccess;
  e = set_rows_smem<8192, true> ();
  if (e == cudaSuccess) e = set_rows_smem<4096, true> ();
  // the single-kernel transforms of the float voltage path (the no-alloc
  // entry point's)
  if (e == cudaSuccess) e = fused_setup<4096, IN_FLOAT, OUT_VOLTAGE, 1> ();
  if (e == cudaSuccess) e = fused_setup<8192, IN_FLOAT, OUT_VOLTAGE, 1> ();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute (k_fwd_cols_fb64<IN_INT8, false>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (FBC_SMEM));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute (k_fwd_cols_fb64<IN_INT8, true>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (FBC_SMEM));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute (k_fwd_cols_fb64<IN_INT16, false>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (FBC_SMEM));
  if (e == cudaSuccess) attr_done.fetch_or (bit);
  return e;
}

cudaError_t launch_convolution (const ConvShape& sh, const ConvTables& tb, const InputView& in,
                                uint64_t part0, unsigned nbatch, float2* scratch, int mode,
                                const FoldView& fv, const VoltView& vv, cudaStream_t st,
                                const KernelClock* clk)
{
  if (nbatch == 0) return cudaSuccess;
  if (sh.n1 == 1)
  {
    switch (sh.nfft)
    {
      case 4096: return run_fused<4096> (sh, tb, in, part0, nbatch, mode, fv, vv, st, clk);
      case 8192: return run_fused<8192> (sh, tb, in, part0, nbatch, mode, fv, vv, st, clk);
      default: return cudaErrorInvalidValue;
    }
  }
  {
    const cudaError_t e = convolution_kernel_setup ();
    if (e != cudaSuccess) return e;
  }
  switch (sh.n1)
  {
    case 2: return run_fourstep_n1<2> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 4: return run_fourstep_n1<4> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 8: return run_fourstep_n1<8> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 16: return run_fourstep_n1<16> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 32: return run_fourstep_n1<32> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    default: return cudaErrorInvalidValue;
  }
}

} // namespace b200
