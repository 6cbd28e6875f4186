// big_cols.cuh -- column passes of 64 .. 512 points, two polarisations
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"
#include "fwd_cols_pair.cuh"

namespace b200 {

namespace {

// Columns of N1 = 32 M points (M = 2 .. 16) with 32 points per thread, M
// threads per column: thread t holds x[t + M r]; a 32-point DFT over r, the
// twiddle w_N1^(t q), one exchange through shared memory, then 32 / M M-point
// DFTs give X[q + 32 p], q = t + M i, in v[i * M + p].  Threads run along the
// columns first, so that global accesses are rows of COLS adjacent values and
// go straight from and to registers; the exchange [q][t][column] is free of
// bank conflicts the same way.  Sixteen points per thread in three passes
// moved every value through shared memory eight times (1438 us forward and
// 1809 us inverse for C2's 2^22-point transforms), this twice: 1073 us
// and 1361 us.
template <int N1>
struct BigCols
{
  static constexpr int M = N1 / 32;
  static constexpr int G = 32 / M;
  static constexpr int T = 256;
};

template <int N1, int COLS>
__device__ __forceinline__ void big_table (float2* tw, const float2* __restrict__ tw1024)
{
  constexpr int M = BigCols<N1>::M;
  for (int i = threadIdx.x; i < N1; i += BigCols<N1>::T)
    tw[i] = __ldg (tw1024 + (i / M) * (i % M) * (1024 / N1) % 1024);
}

// x: the column's exchange area, [q][t] COLS apart; every thread of the block
// calls it (two block barriers, the first after the caller's last use of x)
template <int N1, int COLS, int D>
__device__ __forceinline__ void big_dft (CP* v, float2* x, const float2* tw, int t)
{
  constexpr int M = BigCols<N1>::M;
  dft::run<32, D> (v);
  __syncthreads ();
#pragma unroll
  for (int q = 0; q < 32; q++)
  {
    const float2 w = tw[q * M + t];
    x[(q * M + t) * COLS] = !q ? v[q].z : D < 0 ? cmul (v[q].z, w) : cmulc (v[q].z, w);
  }
  __syncthreads ();
#pragma unroll
  for (int i = 0; i < BigCols<N1>::G; i++)
  {
#pragma unroll
    for (int s = 0; s < M; s++) v[i * M + s].z = x[((t + M * i) * M + s) * COLS];
    dft::run<M, D> (v + i * M);
  }
}

template <int N1> constexpr size_t fwd_big_smem () { return size_t (8192 + N1) * sizeof (float2); }

// one polarisation of unpack_pair
template <int KIND, bool AFFINE>
__device__ __forceinline__ float2 unpack_one (typename RawPair<KIND>::T w, int p, const UnpackPair& u)
{
  if constexpr (KIND == IN_INT16)
  {
    const C2 x = unpack_pair<KIND, AFFINE> (make_uint2 (p ? w.y : w.x, 0), u);
    return make_float2 (x.re.x, x.im.x);
  }
  else
  {
    const C2 x = unpack_pair<KIND, AFFINE> (w >> (16 * p), u);
    return make_float2 (x.re.x, x.im.x);
  }
}

// Forward: unpack (and window) on load, the four-step twiddle w_N^{k1 i2}, rows
// of the scratch out, one polarisation after the other (the raw words are
// read again for the second: kept, they spill).
template <int N1, int KIND, bool AFFINE>
__global__ void __launch_bounds__ (256, 2)
k_fwd_cols_big_pair (const InputView in, const float* __restrict__ lut, const uint64_t step,
                     const uint64_t part0, const unsigned n2, const float2* __restrict__ tw4,
                     const float2* __restrict__ tw1024, float2* __restrict__ scratch,
                     const float* __restrict__ apod)
{
  using B = BigCols<N1>;
  constexpr int M = B::M, COLS = B::T / M;
  extern __shared__ __align__ (16) float2 s_big[];
  float2* tw = s_big + 8192;
  __shared__ float s_lut[KIND == IN_INT8 && !AFFINE ? 256 : 1];
  if (KIND == IN_INT8 && !AFFINE) load_lut (in, lut, s_lut);
  big_table<N1, COLS> (tw, tw1024);
  __syncthreads ();
  const UnpackPair u {s_lut, in.lut_scale, in.offset_binary ? 0u : 0x80008000u};
  const int j = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const unsigned i2 = blockIdx.x * COLS + j;
  const unsigned b = blockIdx.y, c = blockIdx.z;
  const uint64_t N = uint64_t (N1) * n2;
  const uint64_t tstep = KIND == IN_FLOAT ? 1 : in.nchan;
  // the block's window lies in one segment of the input (the carried prefix
  // or the main block) except where a part straddles the prefix's end
  const uint64_t ta = (part0 + b) * step + i2, tb0 = ta - j;
  const bool in_pre = tb0 < in.npre;
  const bool one = !in_pre || tb0 + uint64_t (N1 - 1) * n2 + COLS - 1 < in.npre;
  // sample t + M r of the column: its segment of the input and place in it
  const auto at = [&] (uint64_t t_of, int r, const void*& base, uint64_t& span) {
    const uint64_t tt = t_of + uint64_t (t + M * r) * n2;
    const bool pre = one ? in_pre : tt < in.npre;
    base = pre ? in.pre : in.main;
    span = pre ? in.pre_span : in.main_span;
    return pre ? tt : tt - in.npre;
  };
#pragma unroll 1
  for (int p = 0; p < 2; p++)
  {
    // opaque to the compiler, which would otherwise keep the tables' values of
    // the first polarisation in registers (and spill) for the second
    const float2* twp = tw;
    const float2* w4 = tw4 + uint64_t (t) * n2 + i2;
    uint64_t tp = ta;
    asm volatile ("" : "+l"(twp), "+l"(w4), "+l"(tp));
    CP v[32];
#pragma unroll
    for (int r = 0; r < 32; r++)
    {
      const void* base;
      uint64_t span;
      const uint64_t tt = at (tp, r, base, span);
      if constexpr (KIND == IN_FLOAT)
        v[r].z = __ldg (static_cast<const float2*> (base) + (uint64_t (c) * 2 + p) * span + tt);
      else
        v[r].z = unpack_one<KIND, AFFINE> (load_pair<KIND> (base, tt * tstep + c, span), p, u);
    }
    if (apod)
    {
      // Apodization::operate on the part before the forward FFT (Convolution.C:739-743)
#pragma unroll
      for (int r = 0; r < 32; r++)
      {
        const float a = __ldg (apod + uint64_t (t + M * r) * n2 + i2);
        v[r].z = make_float2 (__fmul_rn (v[r].z.x, a), __fmul_rn (v[r].z.y, a));
      }
    }
    big_dft<N1, COLS, -1> (v, s_big + j, twp, t);
    // (row 0 of the twiddle table is 1)
    float2* dst = scratch + ((uint64_t (b) * in.nchan + c) * 2 + p) * N + uint64_t (t) * n2 + i2;
#pragma unroll
    for (int i = 0; i < B::G; i++)
#pragma unroll
      for (int s = 0; s < M; s++)
      {
        const unsigned o = (M * i + 32 * s) * n2;
        dst[o] = cmul (v[i * M + s].z, __ldg (w4 + o));
      }
  }
}

template <int N1, int NOUT> struct InvBig
{
  using RF = RowFold<NOUT, 4>;
  static constexpr int COLS = 128 / BigCols<N1>::M;
};

template <int N1> constexpr size_t inv_big_smem () { return size_t (8192 + N1) * sizeof (float2); }

// Inverse columns of the During filterbank: half the threads take each
// polarisation; the columns of a block lie in one output channel's segment
// (seg >= 64).  The two hand each other half their samples through the
// exchange area, after which every thread detects 16 samples.
template <int N1, int MODE, int NOUT, bool LONG>
__global__ void __launch_bounds__ (256, 2)
k_inv_cols_big_pair (const float2* __restrict__ scratch, const DuringShape sh, const uint64_t part0,
                     const float2* __restrict__ twd, const float2* __restrict__ tw1024,
                     const FoldView fv, const VoltView vv)
{
  using B = BigCols<N1>;
  using RF = typename InvBig<N1, NOUT>::RF;
  constexpr int M = B::M, COLS = InvBig<N1, NOUT>::COLS, H = 128;     // threads per polarisation
  extern __shared__ __align__ (16) float2 s_big[];
  float2* tw = s_big + 8192;
  __shared__ __align__ (16) float s_fold[LONG ? 8 * RF::WORDS : 4];
  big_table<N1, COLS> (tw, tw1024);
  const int pol = threadIdx.x / H, j = threadIdx.x % COLS, t = threadIdx.x % H / COLS;
  const unsigned i0 = blockIdx.x * COLS, i2 = i0 + j;
  const unsigned b = blockIdx.y, cin = blockIdx.z;
  const uint64_t N = uint64_t (N1) * sh.n2;
  const unsigned c = cin * sh.nsub + i0 / sh.seg, t2 = i2 % sh.seg;
  const float2* src = scratch + ((uint64_t (b) * sh.nchan_in + cin) * 2 + pol) * N + i2;
  CP v[32];
#pragma unroll
  for (int r = 0; r < 32; r++) v[r].z = __ldcs (src + uint64_t (t + M * r) * sh.n2);
#pragma unroll
  for (int r = 0; r < 32; r++)
  {
    // exp(+2 pi i k1 t2 / freq_res); the table's row 0 is 1
    v[r].z = cmulc (v[r].z, __ldg (twd + uint64_t (t + M * r) * sh.seg + t2));
  }
  big_dft<N1, COLS, +1> (v, s_big + pol * 4096 + j, tw, t);
  __syncthreads ();                    // the exchange has been read
  // the profile columns of the thread's samples, asked for together
  const uint64_t tbase = (part0 + b) * sh.nkeep;
  const auto local_time = [&] (int m) {
    return uint64_t (t + M * (m / (M / 2)) + 32 * (2 * (m % (M / 2)) + pol)) * sh.seg + t2;
  };
  unsigned fcol[MODE == OUT_FOLD ? 16 : 1];
  if constexpr (MODE == OUT_FOLD)
  {
#pragma unroll
    for (int m = 0; m < 16; m++)
    {
      const uint64_t tl = local_time (m);
      const bool ok = tl >= sh.nfilt_pos && tl < sh.nfilt_pos + sh.nkeep;
      fcol[m] = fold_column (fv, ok, tbase + (tl - sh.nfilt_pos));
    }
  }
  // samples p even stay with polarisation 0, p odd with polarisation 1
  float2* x = s_big + pol * 2048 + threadIdx.x % H;
#pragma unroll
  for (int i = 0; i < B::G; i++)
#pragma unroll
    for (int s = 0; s < M / 2; s++)
    {
      const int e = i * M + 2 * s, m = i * (M / 2) + s;
      x[m * H] = pol ? v[e].z : v[e + 1].z;
      v[m].z = pol ? v[e + 1].z : v[e].z;
    }
  __syncthreads ();
  const float2* y = s_big + (pol ^ 1) * 2048 + threadIdx.x % H;
  RF rf (s_fold + (LONG ? (threadIdx.x >> 5) * RF::WORDS : 0),
         fv.profiles + uint64_t (c) * NOUT * fv.stride, fv.stride, c == 0 ? fv.hits : nullptr);
#pragma unroll
  for (int m = 0; m < 16; m++)
  {
    const float2 z = y[m * H];
    const float2 pv = pol ? z : v[m].z, qv = pol ? v[m].z : z;
    if constexpr (MODE == OUT_VOLTAGE)
    {
      const uint64_t tl = local_time (m);
      if (tl >= sh.nfilt_pos && tl < sh.nfilt_pos + sh.nkeep)
      {
        float2* o = vv.out + uint64_t (c) * 2 * vv.span + tbase + (tl - sh.nfilt_pos);
        o[0] = pv;
        o[vv.span] = qv;
      }
    }
    else
    {
      detect_row<LONG> (rf, fv.state, 2, fcol[m], pv, qv);
      if (LONG && (m + 1) % RF::ROWS == 0) rf.flush ();
    }
  }
}

template <int N1, int KIND, bool AFFINE>
cudaError_t launch_fwd_big_pair_t (const DuringShape& sh, const DuringTables& tb,
                                   const InputView& in, uint64_t part0, unsigned nbatch,
                                   float2* scratch, cudaStream_t st)
{
  auto k = k_fwd_cols_big_pair<N1, KIND, AFFINE>;
  const cudaError_t e = cudaFuncSetAttribute (k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              int (fwd_big_smem<N1> ()));
  if (e != cudaSuccess) return e;
  const dim3 grid (sh.n2 / (256 / BigCols<N1>::M), nbatch, sh.nchan_in);
  k<<<grid, 256, fwd_big_smem<N1> (), st>>> (in, tb.lut, sh.in_step, part0, sh.n2, tb.tw4,
                                             tb.tw1024, scratch, tb.apod);
  return cudaGetLastError ();
}

// two polarisations in aligned words (fwd_pair_aligned)
template <int N1>
cudaError_t launch_fwd_big_pair (const DuringShape& sh, const DuringTables& tb, const InputView& in,
                                 uint64_t part0, unsigned nbatch, float2* scratch, cudaStream_t st)
{
  if (in.kind == IN_INT8 && in.lut_scale != 0.f)
    return launch_fwd_big_pair_t<N1, IN_INT8, true> (sh, tb, in, part0, nbatch, scratch, st);
  if (in.kind == IN_INT8)
    return launch_fwd_big_pair_t<N1, IN_INT8, false> (sh, tb, in, part0, nbatch, scratch, st);
  if (in.kind == IN_INT16)
    return launch_fwd_big_pair_t<N1, IN_INT16, false> (sh, tb, in, part0, nbatch, scratch, st);
  return launch_fwd_big_pair_t<N1, IN_FLOAT, false> (sh, tb, in, part0, nbatch, scratch, st);
}

template <int N1, int MODE, int NOUT>
cudaError_t launch_inv_big_pair (const DuringShape& sh, const DuringTables& tb, uint64_t part0,
                                 unsigned nbatch, const float2* scratch, const FoldView& fv,
                                 const VoltView& vv, cudaStream_t st)
{
  auto k = MODE == OUT_FOLD && fv.long_bins ? k_inv_cols_big_pair<N1, MODE, NOUT, MODE == OUT_FOLD>
                                            : k_inv_cols_big_pair<N1, MODE, NOUT, false>;
  const cudaError_t e = cudaFuncSetAttribute (k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              int (inv_big_smem<N1> ()));
  if (e != cudaSuccess) return e;
  const dim3 grid (sh.n2 / InvBig<N1, NOUT>::COLS, nbatch, sh.nchan_in);
  k<<<grid, 256, inv_big_smem<N1> (), st>>> (scratch, sh, part0, tb.twd, tb.tw1024, fv, vv);
  return cudaGetLastError ();
}

} // namespace

} // namespace b200
