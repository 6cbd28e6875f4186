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
#include "fb64_cols.cuh"
#include "fwd_cols_pair.cuh"
#include "inv_cols_split.cuh"
#include "rows32.cuh"
#include "rows64.cuh"

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
    StockhamPass<N, R, T, D>::load (threadIdx.x % T, s, v);
    __syncthreads ();
    StockhamPass<N, R, T, D>::compute_store (threadIdx.x % T, Ns, v, s, tw);
    __syncthreads ();
    smem_pass<N, T, D, P + 1> (s, v, tw);
  }
}

// N-point FFT of s[spad(0..N-1)] in place by T threads; the caller has
// synchronised after writing s.  Returns synchronised.  Groups of T threads may
// transform their own arrays side by side (the barriers are the block's).
template <int N, int T, int D>
__device__ __forceinline__ void smem_fft (float2* s, const float2* tw)
{
  float2 v[N / T];
  smem_pass<N, T, D, 0> (s, v, tw);
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

// Groups of T threads take one polarisation each, side by side or one after the
// other.  Side by side (4096 points; 8192 do not fit 512 threads) a block is
// done sooner but alone on its SM; one after the other two blocks share an SM
// and overlap each other's barriers.  In blocks per SM, rounded up, and us
// (voltages of two polarisations, one after the other / side by side): 1:
// 28.6 / 24.5, 2: 36.9 / 40.9, 3: 61.4 / 57.3 (444 blocks of a fold: 105 / 91),
// 4: 67.6 / 73.8, 27: 418 / 469.
template <int T>
constexpr unsigned fused_groups (unsigned npol, unsigned blocks, unsigned nsm)
{
  const unsigned per_sm = (blocks + nsm - 1) / nsm;
  return 2 * T <= 512 && (per_sm == 1 || per_sm == 3) ? npol : 1;
}

template <int N, int T, int KIND, int MODE, int NOUT>
__global__ void __launch_bounds__ (512, 1)
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
  const unsigned groups = blockDim.x / T, group = threadIdx.x / T, tid = threadIdx.x % T;
  load_lut (in, lut, s_lut);
  __syncthreads ();
  const float2* h = H + uint64_t (c) * N;
  for (unsigned p = group; p < npol; p += groups)
  {
    float2* sp = s + p * SP;
#pragma unroll 4
    for (int i = tid; i < N; i += T)
    {
      float2 x = fetch<KIND> (in, s_lut, c, p, part * nkeep + i);
      if (apod)
      {
        const float w = __ldg (apod + i);
        x = make_float2 (__fmul_rn (x.x, w), __fmul_rn (x.y, w));
      }
      sp[spad (i)] = x;
    }
    __syncthreads ();
    smem_fft<N, T, -1> (sp, tw);
#pragma unroll 4
    for (int i = tid; i < N; i += T)
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
  const unsigned rounds = unsigned ((nkeep + blockDim.x - 1) / blockDim.x);
  for (unsigned r = 0; r < rounds; r++)
  {
    const uint64_t j = uint64_t (r) * blockDim.x + threadIdx.x;
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
  // voltages need no exchange of the polarisations: 2^17-point transforms of
  // 2 M samples in 20.7 us against 25.0
  if constexpr (N1 >= 8 && NPOL == 2 && MODE != OUT_VOLTAGE)
  {
    launch_inv_split<N1, NOUT> (scratch, {sh.n2, sh.n2, sh.nchan, sh.nkeep, sh.nfilt_pos}, part0,
                                grid.y, tb.tw4, tb.nsm, fv, st);
    return;
  }
  else
  {
  if (N1 == 32) grid.x = sh.n2 / 64;        // two threads per column
  k_inv_cols<N1, NPOL, MODE, NOUT><<<grid, 128, 0, st>>> (scratch, sh.n2, sh.nchan, sh.nkeep,
                                                          sh.nfilt_pos, part0, tb.tw4, fv, vv);
  }
}

// 4096-point rows: k_rows64.  8192-point rows: k_rows32, or k_rows_mma when
// the tensor-core arithmetic is asked for.
void launch_rows (unsigned nrows, float2* scratch, const ConvTables& tb, unsigned n1,
                  const ConvShape& sh, cudaStream_t st)
{
  if (sh.n2 == 4096)
  {
    launch_rows64 (nrows, scratch, tb.H, n1, sh.nchan, sh.npol, tb.nsm, tb.err, st);
    return;
  }
  if (tb.tc_splits)
  {
    launch_rows_mma (nrows, scratch, tb, n1, sh, st);
    return;
  }
  // persistent: as many CTAs as are resident at once
  const unsigned grid = std::min<unsigned> (nrows, rows32_ctas_per_sm<8192> () * unsigned (tb.nsm));
  k_rows32<8192, true><<<grid, Row32<8192>::T, rows32_smem_bytes<8192> (), st>>> (
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
    if ((N1 != 8 && N1 != 16) || in.fb_nsub != 64 || sh.nchan != 64 || in.nchan != 1
        || in.npol != 2 || sh.npol != 2 || tb.apod || (in.kind != IN_INT8 && in.kind != IN_INT16))
      return cudaErrorInvalidValue;
    ClockScope cs (clk, KK_FWD_COLS, st);
    if constexpr (N1 == 8 || N1 == 16)
      launch_fb64<N1> (in, tb.lut, sh.nkeep, part0, nbatch, sh.n2, tb.tw4, scratch, st);
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
  if (sh.n2 != 8192 && sh.n2 != 4096) return cudaErrorInvalidValue;
  launch_rows (nrows, scratch, tb, N1, sh, st);
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
  const unsigned groups = fused_groups<T> (in.npol, nbatch * sh.nchan, unsigned (tb.nsm));
  kern<<<dim3 (nbatch, sh.nchan), T * groups, smem, st>>> (
      in, tb.lut, tb.tw2, tb.H, sh.nkeep, sh.nfilt_pos, part0, fv, vv, tb.apod);
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
  return n2 == 8192 ? rows32_ctas_per_sm<8192> () : unsigned (R64_GROUPS);
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
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute (k_rows64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int (R64_SMEM));
  // the single-kernel transforms of the float voltage path (the no-alloc
  // entry point's)
  if (e == cudaSuccess) e = fused_setup<4096, IN_FLOAT, OUT_VOLTAGE, 1> ();
  if (e == cudaSuccess) e = fused_setup<8192, IN_FLOAT, OUT_VOLTAGE, 1> ();
  if (e == cudaSuccess) e = fb64_setup ();
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
