// during.cu -- the filterbank with a response (FilterbankEngineCPU.C:379-535)

#include "big_cols.cuh"
#include "fwd_cols.cuh"
#include "fwd_cols_pair.cuh"
#include "inv_cols_split.cuh"
#include "rows32.cuh"

namespace b200 {

namespace {

// --------------------------------------------------------------------------
// Filterbank with a response ("During")
// --------------------------------------------------------------------------

// Barrier of a group of TS consecutive threads that exchange data only among
// themselves: a warp barrier when the group lies inside one warp (TS divides
// 32), else the block's.
template <int TS>
__device__ __forceinline__ void group_sync ()
{
  static_assert (TS <= 32 ? 32 % TS == 0 : TS % 32 == 0, "groups must tile the warps");
  if constexpr (TS <= 32)
    __syncwarp ();
  else
    __syncthreads ();
}

// One radix pass of an N-point transform run by the stockham_threads(N)
// threads of one group (lane = index in the group), both sides in the padded
// layout relative to the group's base, or the output unpadded (PO false).
// Every thread of the block calls it.  Its barriers cover the group only, so
// a caller that reads or writes the groups' buffers across groups puts a
// block barrier between that and the passes.
template <int N, int D, int P, bool PO>
__device__ __forceinline__ void gpass (int lane, const float2* src, float2* dst, float2* v,
                                       const float2* tab)
{
  if constexpr (P < stockham_npass (N))
  {
    constexpr int T = stockham_threads (N);
    constexpr int R = stockham_radix (N, P);
    constexpr int Ns = stockham_ns (N, P);
    StockhamPassT<N, R, T, D, true, PO>::load (lane, src, v);
    group_sync<T> ();
    StockhamPassT<N, R, T, D, true, PO>::compute_store (
        lane, Ns, v, dst, P ? tab + pass_table_offset (N, P) : nullptr);
    group_sync<T> ();
  }
}

constexpr int DUR_N2 = 8192;

template <int SEG>
constexpr size_t during_rows_smem ()
{
  return size_t (spad_size (DUR_N2) + Row32<DUR_N2>::TABN + pass_tables_size (SEG))
         * sizeof (float2);
}

// Rows of the big transform (persistent CTAs, one row at a time, two per SM):
// the forward n2-point FFT with 32 points per thread in three passes
// (Row32), the response of each output channel on its segment multiplied in
// registers (Response::operate over nchan_subband channels from
// input_ichan*nchan_subband, FilterbankEngineCPU.C:480-484), then the
// seg-point inverse FFT of every segment, written back in place: each group
// of seg/16 threads takes two segments.  Row r of the scratch is row
// k1 = r mod n1 of (part, input channel, pol).
template <int SEG>
__global__ void __launch_bounds__ (Row32<DUR_N2>::T, 2)
k_rows_during (float2* __restrict__ scratch, const float2* __restrict__ ptab_seg,
               const float2* __restrict__ H, const unsigned n1, const unsigned nsub,
               const unsigned npol, const unsigned nchan_in, const unsigned nrows,
               const unsigned inner)
{
  constexpr int N2 = DUR_N2;
  using RS = Row32<N2>;
  constexpr int T = RS::T;
  constexpr int TABS = pass_tables_size (SEG);
  constexpr int TS = stockham_threads (SEG);
  constexpr int NPS = stockham_npass (SEG);
  constexpr int NG = T / TS;                      // segment groups
  constexpr unsigned ROW_BYTES = N2 * sizeof (float2);
  constexpr unsigned CHUNK = 16384;
  static_assert (NPS == 2 || NPS == 3, "segment transforms of 64 .. 4096 points");
  static_assert (T % TS == 0 && (N2 / SEG) == 2 * NG, "each group takes two segments");
  extern __shared__ __align__ (16) float2 s_dur[];
  float2* work = s_dur;
  float2* tab1 = work + spad_size (N2);
  float2* th = tab1 + RS::TAB1;
  float2* tl = th + RS::TABH;
  float2* tabs = tab1 + RS::TABN;
  const int tid = threadIdx.x;
  for (int i = tid; i < RS::TABN; i += T) tab1[i] = RS::table_entry (i);
  for (int i = tid; i < TABS; i += T) tabs[i] = __ldg (ptab_seg + i);
  const int g = tid / TS, lane = tid % TS;
  // As in k_rows32: rows walked with their response rows (input channel,
  // k1) outermost, parts and polarisations innermost (inner of them), each
  // CTA a contiguous run, the response kept in L1 (evict-last loads) and the
  // scratch rows streamed (evict-first).
  const auto row_of = [=] (unsigned idx, unsigned& hrow) {
    hrow = idx / inner;                             // cin * n1 + k1
    const unsigned bp = idx % inner;
    return ((bp / npol) * nchan_in * n1 + hrow / n1 * n1) * npol + (bp % npol) * n1 + hrow % n1;
  };
  float2 v[32];
  const unsigned run = (nrows + gridDim.x - 1) / gridDim.x;
  const unsigned idx_end = min (nrows, (blockIdx.x + 1) * run);
  for (unsigned idx = blockIdx.x * run; idx < idx_end; idx++)
  {
    unsigned hrow = 0;
    const unsigned row = row_of (idx, hrow);
    const unsigned k1 = hrow % n1;
    const unsigned cin = hrow / n1;
    float2* grow = scratch + uint64_t (row) * N2;
    if (tid == 0 && idx + 1 < idx_end)
    {
      unsigned nh = 0;
      const char* nr = reinterpret_cast<const char*> (scratch + uint64_t (row_of (idx + 1, nh)) * N2);
      for (unsigned o = 0; o < ROW_BYTES; o += CHUNK) prefetch_l2 (nr + o, CHUNK);
    }
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int r = 0; r < 16; r++) v[16 * b + r] = __ldcs (grow + tid + b * T + r * RS::NS2);
    __syncthreads ();     // the previous row's segment passes are done
    RS::template p0_compute_store<-1> (tid, v, work);
    __syncthreads ();
    RS::p1_load (tid, work, v);
    __syncthreads ();
    RS::template p1_compute_store<-1> (tid, v, work, tab1);
    __syncthreads ();
    RS::p2_load (tid, work, v);
    __syncthreads ();
    RS::template p2_compute<-1> (tid, v, th, tl);
    // position i = cs*SEG + f2 of row k1 is bin k1 + n1*f2 of output channel
    // cin*nsub + cs: (f_r d_r - f_i d_i, f_i d_r + f_r d_i), Response.C:662-726
    const float2* hc = H + (uint64_t (cin) * nsub * n1 + k1) * SEG;
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int r = 0; r < 16; r++)
      {
        const int i = tid + b * T + r * RS::NS2;
        const unsigned cs = unsigned (i) / SEG, f2 = unsigned (i) % SEG;
        const float2 f = ldg_evict_last (hc + uint64_t (cs) * n1 * SEG + f2);
        const float2 d = v[16 * b + r];
        work[spad (i)] = make_float2 (d.x * f.x - d.y * f.y, d.x * f.y + d.y * f.x);
      }
    __syncthreads ();
    // spad(s*SEG + i) = spad(s*SEG) + spad(i) because SEG is a multiple of 16
#pragma unroll
    for (int s2 = 0; s2 < 2; s2++)
    {
      const int sg = g + s2 * NG;
      float2* wseg = work + spad (sg * SEG);
      float2* gseg = grow + sg * SEG;
      if constexpr (NPS == 2)
      {
        gpass<SEG, +1, 0, true> (lane, wseg, wseg, v, tabs);
        gpass<SEG, +1, 1, false> (lane, wseg, gseg, v, tabs);
      }
      else
      {
        gpass<SEG, +1, 0, true> (lane, wseg, wseg, v, tabs);
        gpass<SEG, +1, 1, true> (lane, wseg, wseg, v, tabs);
        gpass<SEG, +1, 2, false> (lane, wseg, gseg, v, tabs);
      }
    }
  }
}

// Inverse column DFTs of the freq_res-point transforms: thread i2 holds
// sample t2 = i2 mod seg of output channel cin*nsub + i2/seg; conjugate
// twiddle exp(+2 pi i k1 t2 / freq_res), n1-point inverse DFT giving samples
// t2 + seg*t1, then the discard of nfilt_pos / nfilt_neg
// (FilterbankEngineCPU.C:516-523) and voltages out, or detection + fold.
// seg >= 64, so the 32 lanes of a warp share one output channel.
template <int N1, int NPOL, int MODE, int NOUT>
__global__ void __launch_bounds__ (128, N1 >= 32 ? 3 : 4)
k_inv_cols_during (const float2* __restrict__ scratch, const DuringShape sh, const uint64_t part0,
                   const float2* __restrict__ twd, const FoldView fv, const VoltView vv)
{
  const unsigned i2 = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned b = blockIdx.y;
  const unsigned cin = blockIdx.z;
  const uint64_t N = uint64_t (N1) * sh.n2;
  const unsigned cs = i2 / sh.seg, t2 = i2 % sh.seg;
  const unsigned c = cin * sh.nsub + cs;
  float* prof = fv.profiles + uint64_t (c) * NOUT * fv.stride;
  unsigned* hits = c == 0 ? fv.hits : nullptr;
  float2 w[N1];
#pragma unroll
  for (int k = 1; k < N1; k++)
    w[k] = __ldg (twd + uint64_t (k) * sh.seg + t2);
  float2 v[NPOL][N1];
#pragma unroll
  for (int p = 0; p < NPOL; p++)
  {
    const float2* src = scratch + ((uint64_t (b) * sh.nchan_in + cin) * NPOL + p) * N + i2;
#pragma unroll
    for (int k = 0; k < N1; k++)
      v[p][k] = src[uint64_t (k) * sh.n2];
#pragma unroll
    for (int k = 1; k < N1; k++)
      v[p][k] = cmulc (v[p][k], w[k]);
    RegDFT<N1, +1>::run (v[p]);
  }
  const uint64_t tbase = (part0 + b) * sh.nkeep;
#pragma unroll
  for (int k = 0; k < N1; k++)
  {
    const uint64_t tl = uint64_t (k) * sh.seg + t2;
    const bool ok = tl >= sh.nfilt_pos && tl < sh.nfilt_pos + sh.nkeep;
    const uint64_t t = tbase + (tl - sh.nfilt_pos);
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
      detect_fold<NOUT> (fv, NPOL, fold_column (fv, ok, t), v[0][k], v[NPOL - 1][k], prof, hits);
  }
}

// Column passes of N1 = 64 .. 512 points (big transforms of up to 2^22 =
// 512 x 8192 points): a CTA of N1 threads takes COLW = 16 adjacent columns,
// loads them row by row (16 consecutive samples per row) into shared memory,
// one column per group of N1/16 threads, and runs the N1-point Stockham
// transforms there (per-pass tables in shared memory).  Column stride
// spad_size(N1) + 1 keeps the 16 columns of a row on different banks.
constexpr int COLW = 16;

// Buffer stride: with 16 columns per CTA (a half-warp touches one row) 1 mod
// 16 float2 keeps the columns on distinct bank pairs; with 8 (a half-warp
// touches two adjacent rows, k even and k + 1) 2 mod 16 does.
template <int N1, int CW = COLW>
B200_CE int colbig_stride () { return spad_size (N1) + (CW >= 16 ? 1 : 2); }

template <int N1>
constexpr size_t colbig_smem ()
{
  return size_t (COLW * colbig_stride<N1> () + pass_tables_size (N1)) * sizeof (float2);
}

// columns per CTA of the inverse pass
template <int N1>
B200_CE int inv_colw () { return N1 >= 512 ? 8 : COLW; }

template <int N1>
constexpr size_t colbig_inv_smem ()
{
  return size_t (inv_colw<N1> () * colbig_stride<N1, inv_colw<N1> ()> () + pass_tables_size (N1))
         * sizeof (float2);
}

// the N1-point transform (direction D) of every column in col[]
template <int N1, int D, int SP = colbig_stride<N1> ()>
__device__ __forceinline__ void colbig_fft (float2* col, const float2* tab)
{
  constexpr int TS = stockham_threads (N1);
  const int g = threadIdx.x / TS, lane = threadIdx.x % TS;
  float2* base = col + g * SP;
  float2 v[16];
  gpass<N1, D, 0, true> (lane, base, base, v, tab);
  gpass<N1, D, 1, true> (lane, base, base, v, tab);
  gpass<N1, D, 2, true> (lane, base, base, v, tab);
}

// Forward: unpack (and window) on load, N1-point DFTs down the columns, the
// four-step twiddle w_N^{k1 i2}, rows of the scratch out.
template <int N1, int KIND>
__global__ void __launch_bounds__ (N1, 1024 / N1)
k_fwd_cols_big (const InputView in, const float* __restrict__ lut, const uint64_t step,
                const uint64_t part0, const unsigned n2, const float2* __restrict__ tw4,
                const float2* __restrict__ ptab_col, float2* __restrict__ scratch,
                const float* __restrict__ apod)
{
  static_assert (stockham_npass (N1) <= 3, "column transforms of at most three passes");
  constexpr int T = N1;
  constexpr int SP = colbig_stride<N1> ();
  constexpr int TAB = pass_tables_size (N1);
  extern __shared__ __align__ (16) float2 s_cb[];
  float2* col = s_cb;
  float2* tab = s_cb + COLW * SP;
  __shared__ float s_lut[256];
  load_lut (in, lut, s_lut);
  for (int i = threadIdx.x; i < TAB; i += T) tab[i] = __ldg (ptab_col + i);
  const unsigned c0 = blockIdx.x * COLW;
  const unsigned b = blockIdx.y;
  const unsigned c = blockIdx.z;
  const uint64_t N = uint64_t (N1) * n2;
  const uint64_t t0 = (part0 + b) * step + c0;
  // thread (kk, j) takes rows k = kk + m KSTEP of column c0 + j
  constexpr int KSTEP = T / COLW;
  const int j = threadIdx.x % COLW, kk = threadIdx.x / COLW;
  // The block's window t0 + k n2 + j lies in one segment of the input (the
  // carried prefix or the main block) except in the parts that straddle the
  // prefix's end; there each sample takes the general fetch.
  const bool one_seg = t0 >= in.npre || t0 + uint64_t (N1 - 1) * n2 + (COLW - 1) < in.npre;
  const bool in_pre = t0 < in.npre;
  const uint64_t ts = in_pre ? t0 : t0 - in.npre;
  const float* ap = apod ? apod + uint64_t (kk) * n2 + c0 + j : nullptr;
  const uint64_t rstep = uint64_t (KSTEP) * n2;
  for (unsigned p = 0; p < in.npol; p++)
  {
    __syncthreads ();
    const auto put = [&] (int k, float2 x) {
      if (ap)
      {
        const float w = __ldg (ap + uint64_t (k - kk) * n2);
        x = make_float2 (__fmul_rn (x.x, w), __fmul_rn (x.y, w));
      }
      col[j * SP + spad (k)] = x;
    };
    if (one_seg && KIND == IN_FLOAT)
    {
      const float2* f = static_cast<const float2*> (in_pre ? in.pre : in.main)
                        + (uint64_t (c) * in.npol + p) * (in_pre ? in.pre_span : in.main_span)
                        + ts + uint64_t (kk) * n2 + j;
      for (int k = kk; k < N1; k += KSTEP, f += rstep) put (k, __ldg (f));
    }
    else if (one_seg)
    {
      // one complex sample per (t, c, p): 2 bytes (int8) or 4 (int16)
      const uint64_t cs = uint64_t (in.nchan) * in.npol;
      const uint64_t i0 = (ts + uint64_t (kk) * n2 + j) * cs + c * in.npol + p;
      const uint64_t istep = rstep * cs;
      if constexpr (KIND == IN_INT8)
      {
        const unsigned short* q = static_cast<const unsigned short*> (in_pre ? in.pre : in.main) + i0;
        for (int k = kk; k < N1; k += KSTEP, q += istep)
        {
          const unsigned short w = __ldg (q);
          put (k, make_float2 (s_lut[w & 0xff], s_lut[w >> 8]));
        }
      }
      else
      {
        const unsigned* q = static_cast<const unsigned*> (in_pre ? in.pre : in.main) + i0;
        for (int k = kk; k < N1; k += KSTEP, q += istep)
        {
          const unsigned w = __ldg (q);
          short re = short (w & 0xffff), im = short (w >> 16);
          if (in.offset_binary)
          {
            re = short (re ^ 0x8000);
            im = short (im ^ 0x8000);
          }
          // SixteenBitUnpacker.C:69: float(x) + 0.5
          put (k, make_float2 (__fadd_rn (float (re), 0.5f), __fadd_rn (float (im), 0.5f)));
        }
      }
    }
    else
      for (int k = kk; k < N1; k += KSTEP)
        put (k, fetch<KIND> (in, s_lut, c, p, t0 + uint64_t (k) * n2 + j));
    __syncthreads ();
    colbig_fft<N1, -1> (col, tab);
    __syncthreads ();                  // the output below reads across columns' groups
    float2* dst = scratch + ((uint64_t (b) * in.nchan + c) * in.npol + p) * N + c0 + j
                  + uint64_t (kk) * n2;
    const float2* tw = tw4 + uint64_t (kk) * n2 + c0 + j;
    for (int k1 = kk; k1 < N1; k1 += KSTEP, dst += rstep, tw += rstep)
    {
      float2 y = col[j * SP + spad (k1)];
      if (k1) y = cmul (y, __ldg (tw));
      *dst = y;
    }
  }
}

// Inverse columns of the During filterbank for N1 = 64 .. 512 and one
// polarisation (two: k_inv_cols_big_pair): the columns of a CTA lie in one output
// channel's segment (seg >= 64); they are loaded with the conjugate twiddle
// exp(+2 pi i k1 t2 / freq_res), transformed, and read back in time order (16
// consecutive samples per row) for the discard and the voltages or detection
// + fold.
template <int N1, int MODE>
__global__ void __launch_bounds__ (inv_colw<N1> () * stockham_threads (N1), 1024 / N1)
k_inv_cols_during_big (const float2* __restrict__ scratch, const DuringShape sh,
                       const uint64_t part0, const float2* __restrict__ twd,
                       const float2* __restrict__ ptab_col, const FoldView fv, const VoltView vv)
{
  constexpr int CW = inv_colw<N1> ();
  constexpr int T = CW * stockham_threads (N1);
  constexpr int SP = colbig_stride<N1, CW> ();
  constexpr int TAB = pass_tables_size (N1);
  extern __shared__ __align__ (16) float2 s_cb[];
  float2* tab = s_cb + CW * SP;
  for (int i = threadIdx.x; i < TAB; i += T) tab[i] = __ldg (ptab_col + i);
  const unsigned c0 = blockIdx.x * CW;
  const unsigned b = blockIdx.y;
  const unsigned cin = blockIdx.z;
  const uint64_t N = uint64_t (N1) * sh.n2;
  const unsigned cs = c0 / sh.seg, t20 = c0 % sh.seg;
  const unsigned c = cin * sh.nsub + cs;
  // thread (kk, j) takes rows k1 = kk + m KSTEP of column c0 + j
  constexpr int KSTEP = T / CW;
  {
    const int j = threadIdx.x % CW, kk = threadIdx.x / CW;
    const float2* src = scratch + (uint64_t (b) * sh.nchan_in + cin) * N + c0 + j
                        + uint64_t (kk) * sh.n2;
    const float2* tw = twd + uint64_t (kk) * sh.seg + t20 + j;
    const uint64_t sstep = uint64_t (KSTEP) * sh.n2, tstep = uint64_t (KSTEP) * sh.seg;
    for (int k1 = kk; k1 < N1; k1 += KSTEP, src += sstep, tw += tstep)
    {
      float2 x = *src;
      if (k1) x = cmulc (x, __ldg (tw));
      s_cb[j * SP + spad (k1)] = x;
    }
  }
  __syncthreads ();
  colbig_fft<N1, +1, SP> (s_cb, tab);
  __syncthreads ();                    // the fold below reads across columns' groups
  const uint64_t tbase = (part0 + b) * sh.nkeep;
  float* prof = fv.profiles + uint64_t (c) * fv.stride;
  unsigned* hits = c == 0 ? fv.hits : nullptr;
  for (int e = threadIdx.x; e < CW * N1; e += T)
  {
    const int j = e % CW, t1 = e / CW;
    const uint64_t tl = uint64_t (t1) * sh.seg + t20 + j;
    const bool ok = tl >= sh.nfilt_pos && tl < sh.nfilt_pos + sh.nkeep;
    const uint64_t t = tbase + (tl - sh.nfilt_pos);
    const float2 v = s_cb[j * SP + spad (t1)];
    if constexpr (MODE == OUT_VOLTAGE)
    {
      if (ok) vv.out[uint64_t (c) * vv.span + t] = v;
    }
    else
      detect_fold<1> (fv, 1, fold_column (fv, ok, t), v, v, prof, hits);
  }
}

} // namespace

namespace {

template <int SEG>
cudaError_t launch_rows_during (unsigned nrows, float2* scratch, const DuringShape& sh,
                                const DuringTables& tb, cudaStream_t st)
{
  constexpr size_t smem = during_rows_smem<SEG> ();
  static_assert (smem <= 227u * 1024u, "row kernel shared memory");
  cudaError_t e = cudaFuncSetAttribute (k_rows_during<SEG>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
  if (e != cudaSuccess) return e;
  // persistent: two CTAs per SM
  const unsigned grid = std::min<unsigned> (nrows, 2 * unsigned (tb.nsm));
  k_rows_during<SEG><<<grid, Row32<DUR_N2>::T, smem, st>>> (
      scratch, tb.ptab_seg, tb.H, sh.n1, sh.nsub, sh.npol, sh.nchan_in, nrows,
      nrows / (sh.n1 * sh.nchan_in));
  return cudaSuccess;
}

template <int N1, int NPOL, int MODE, int NOUT>
void launch_inv_during (const DuringShape& sh, dim3 grid, const float2* scratch, uint64_t part0,
                        const DuringTables& tb, const FoldView& fv, const VoltView& vv,
                        cudaStream_t st)
{
  // voltages need no exchange of the polarisations (calls of 8 M samples, int8,
  // split / a thread per column: 64 x 4096 206.9 / 198.7 us, 64 x 2048 194.6 /
  // 191.5, 32 x 2048 183.3 / 180.3)
  if constexpr (N1 >= 8 && N1 <= 32 && NPOL == 2 && MODE != OUT_VOLTAGE)
    launch_inv_split<N1, NOUT> (scratch, {sh.n2, sh.seg, sh.nchan_in, sh.nkeep, sh.nfilt_pos},
                                part0, grid.y, tb.twd, tb.nsm, fv, st);
  else
    k_inv_cols_during<N1, NPOL, MODE, NOUT><<<grid, 128, 0, st>>> (scratch, sh, part0, tb.twd, fv,
                                                                   vv);
}

template <int N1, int NPOL>
void launch_inv_during_m (const DuringShape& sh, dim3 grid, const float2* scratch,
                          uint64_t part0, const DuringTables& tb, int mode, const FoldView& fv,
                          const VoltView& vv, cudaStream_t st)
{
  if (mode == OUT_VOLTAGE)
    launch_inv_during<N1, NPOL, OUT_VOLTAGE, 1> (sh, grid, scratch, part0, tb, fv, vv, st);
  else if (NPOL == 1 || fv.nout == 1)
    launch_inv_during<N1, NPOL, OUT_FOLD, 1> (sh, grid, scratch, part0, tb, fv, vv, st);
  else if (fv.nout == 2)
    launch_inv_during<N1, NPOL, OUT_FOLD, 2> (sh, grid, scratch, part0, tb, fv, vv, st);
  else
    launch_inv_during<N1, NPOL, OUT_FOLD, 4> (sh, grid, scratch, part0, tb, fv, vv, st);
}

template <int N1>
cudaError_t run_during_n1 (const DuringShape& sh, const DuringTables& tb, const InputView& in,
                           uint64_t part0, unsigned nbatch, float2* scratch, int mode,
                           const FoldView& fv, const VoltView& vv, cudaStream_t st,
                           const KernelClock* clk)
{
  const dim3 gcol (sh.n2 / 128, nbatch, sh.nchan_in);
  const dim3 gfwd (sh.n2 / fwd_cols_per_block<N1> (), nbatch, sh.nchan_in);
  {
    ClockScope cs (clk, KK_FWD_COLS, st);
    if (N1 > 1 && in.npol == 2 && fwd_pair_aligned (in))
    {
      if constexpr (N1 > 1)
        launch_fwd_pair<N1> (in, tb.lut, sh.in_step, part0, nbatch, sh.n2, tb.tw4, scratch, tb.apod,
                             tb.nsm, st);
    }
    else if (in.kind == IN_INT8)
      k_fwd_cols<N1, IN_INT8><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.in_step, part0, sh.n2, tb.tw4,
                                                     scratch, tb.apod);
    else if (in.kind == IN_INT16)
      k_fwd_cols<N1, IN_INT16><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.in_step, part0, sh.n2,
                                                      tb.tw4, scratch, tb.apod);
    else
      k_fwd_cols<N1, IN_FLOAT><<<gfwd, 128, 0, st>>> (in, tb.lut, sh.in_step, part0, sh.n2,
                                                      tb.tw4, scratch, tb.apod);
  }
  const unsigned nrows = N1 * nbatch * sh.nchan_in * sh.npol;
  cudaError_t e = cudaSuccess;
  {
    ClockScope cs (clk, KK_ROWS, st);
    switch (sh.seg)
    {
      case 64: e = launch_rows_during<64> (nrows, scratch, sh, tb, st); break;
      case 128: e = launch_rows_during<128> (nrows, scratch, sh, tb, st); break;
      case 256: e = launch_rows_during<256> (nrows, scratch, sh, tb, st); break;
      case 512: e = launch_rows_during<512> (nrows, scratch, sh, tb, st); break;
      case 1024: e = launch_rows_during<1024> (nrows, scratch, sh, tb, st); break;
      case 2048: e = launch_rows_during<2048> (nrows, scratch, sh, tb, st); break;
      case 4096: e = launch_rows_during<4096> (nrows, scratch, sh, tb, st); break;
      default: return cudaErrorInvalidValue;
    }
  }
  if (e != cudaSuccess) return e;
  ClockScope cs (clk, KK_INV_COLS, st);
  if (sh.npol == 2)
    launch_inv_during_m<N1, 2> (sh, gcol, scratch, part0, tb, mode, fv, vv, st);
  else
    launch_inv_during_m<N1, 1> (sh, gcol, scratch, part0, tb, mode, fv, vv, st);
  return cudaGetLastError ();
}

// two polarisations: k_inv_cols_big_pair; one: k_inv_cols_during_big
template <int N1>
cudaError_t launch_inv_during_big (const DuringShape& sh, dim3 grid, const float2* scratch,
                                   uint64_t part0, const DuringTables& tb, int mode,
                                   const FoldView& fv, const VoltView& vv, cudaStream_t st)
{
  if (sh.npol == 2)
  {
    if (mode == OUT_VOLTAGE)
      return launch_inv_big_pair<N1, OUT_VOLTAGE, 1> (sh, tb, part0, grid.y, scratch, fv, vv, st);
    if (fv.nout == 1)
      return launch_inv_big_pair<N1, OUT_FOLD, 1> (sh, tb, part0, grid.y, scratch, fv, vv, st);
    if (fv.nout == 2)
      return launch_inv_big_pair<N1, OUT_FOLD, 2> (sh, tb, part0, grid.y, scratch, fv, vv, st);
    return launch_inv_big_pair<N1, OUT_FOLD, 4> (sh, tb, part0, grid.y, scratch, fv, vv, st);
  }
  constexpr size_t smem = colbig_inv_smem<N1> ();
  constexpr int T = inv_colw<N1> () * stockham_threads (N1);
  grid.x = sh.n2 / inv_colw<N1> ();
  auto k = mode == OUT_VOLTAGE ? k_inv_cols_during_big<N1, OUT_VOLTAGE>
                               : k_inv_cols_during_big<N1, OUT_FOLD>;
  const cudaError_t e = cudaFuncSetAttribute (k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              int (smem));
  if (e != cudaSuccess) return e;
  k<<<grid, T, smem, st>>> (scratch, sh, part0, tb.twd, tb.ptab_col, fv, vv);
  return cudaGetLastError ();
}

template <int N1>
cudaError_t run_during_big (const DuringShape& sh, const DuringTables& tb, const InputView& in,
                            uint64_t part0, unsigned nbatch, float2* scratch, int mode,
                            const FoldView& fv, const VoltView& vv, cudaStream_t st,
                            const KernelClock* clk)
{
  static_assert (colbig_inv_smem<N1> () <= 227u * 1024u, "column kernel shared memory");
  const dim3 gcol (sh.n2 / COLW, nbatch, sh.nchan_in);
  {
    ClockScope cs (clk, KK_FWD_COLS, st);
    constexpr size_t smem = colbig_smem<N1> ();
    if (in.npol == 2 && fwd_pair_aligned (in))
    {
      const cudaError_t e = launch_fwd_big_pair<N1> (sh, tb, in, part0, nbatch, scratch, st);
      if (e != cudaSuccess) return e;
    }
    else if (in.kind == IN_INT8)
    {
      cudaFuncSetAttribute (k_fwd_cols_big<N1, IN_INT8>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
      k_fwd_cols_big<N1, IN_INT8><<<gcol, N1, smem, st>>> (in, tb.lut, sh.in_step, part0, sh.n2,
                                                          tb.tw4, tb.ptab_col, scratch, tb.apod);
    }
    else if (in.kind == IN_INT16)
    {
      cudaFuncSetAttribute (k_fwd_cols_big<N1, IN_INT16>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
      k_fwd_cols_big<N1, IN_INT16><<<gcol, N1, smem, st>>> (in, tb.lut, sh.in_step, part0, sh.n2,
                                                           tb.tw4, tb.ptab_col, scratch, tb.apod);
    }
    else
    {
      cudaFuncSetAttribute (k_fwd_cols_big<N1, IN_FLOAT>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
      k_fwd_cols_big<N1, IN_FLOAT><<<gcol, N1, smem, st>>> (in, tb.lut, sh.in_step, part0, sh.n2,
                                                           tb.tw4, tb.ptab_col, scratch, tb.apod);
    }
  }
  const unsigned nrows = N1 * nbatch * sh.nchan_in * sh.npol;
  cudaError_t e = cudaSuccess;
  {
    ClockScope cs (clk, KK_ROWS, st);
    switch (sh.seg)
    {
      case 64: e = launch_rows_during<64> (nrows, scratch, sh, tb, st); break;
      case 128: e = launch_rows_during<128> (nrows, scratch, sh, tb, st); break;
      case 256: e = launch_rows_during<256> (nrows, scratch, sh, tb, st); break;
      case 512: e = launch_rows_during<512> (nrows, scratch, sh, tb, st); break;
      case 1024: e = launch_rows_during<1024> (nrows, scratch, sh, tb, st); break;
      case 2048: e = launch_rows_during<2048> (nrows, scratch, sh, tb, st); break;
      case 4096: e = launch_rows_during<4096> (nrows, scratch, sh, tb, st); break;
      default: return cudaErrorInvalidValue;
    }
  }
  if (e != cudaSuccess) return e;
  ClockScope cs (clk, KK_INV_COLS, st);
  return launch_inv_during_big<N1> (sh, gcol, scratch, part0, tb, mode, fv, vv, st);
}

} // namespace

namespace {
__global__ void k_window_response (float2* __restrict__ out, const float2* __restrict__ in,
                                   const float* __restrict__ w, const uint64_t n,
                                   const unsigned n1, const unsigned seg)
{
  const uint64_t idx = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const uint64_t fr = uint64_t (n1) * seg;
  const unsigned r = unsigned (idx % fr);
  const unsigned f = r / seg + n1 * (r % seg);
  const float2 h = in[idx];
  const float x = __ldg (w + f);
  out[idx] = make_float2 (__fmul_rn (h.x, x), __fmul_rn (h.y, x));
}
} // namespace

cudaError_t launch_window_response (float2* out, const float2* in, const float* window,
                                    unsigned nchan, unsigned n1, unsigned seg, cudaStream_t st)
{
  const uint64_t n = uint64_t (nchan) * n1 * seg;
  g_launches++;
  k_window_response<<<unsigned ((n + 255) / 256), 256, 0, st>>> (out, in, window, n, n1, seg);
  return cudaGetLastError ();
}

// (its kernels' shared-memory opt-in goes with each launch)
cudaError_t during_kernel_setup ()
{
  cudaFuncAttributes a;
  return cudaFuncGetAttributes (&a, k_window_response);
}

bool during_supported (unsigned nsub, unsigned freq_res)
{
  if (nsub < 2 || nsub > 128 || (nsub & (nsub - 1))) return false;
  const uint64_t n = uint64_t (nsub) * freq_res;
  return freq_res && (freq_res & (freq_res - 1)) == 0 && n >= 2 * DUR_N2 && n <= 512 * DUR_N2;
}

cudaError_t launch_filterbank_during (const DuringShape& sh, const DuringTables& tb,
                                      const InputView& in, uint64_t part0, unsigned nbatch,
                                      float2* scratch, int mode, const FoldView& fv,
                                      const VoltView& vv, cudaStream_t st,
                                      const KernelClock* clk)
{
  if (nbatch == 0) return cudaSuccess;
  if (!during_supported (sh.nsub, sh.freq_res) || sh.n2 != unsigned (DUR_N2)
      || uint64_t (sh.n1) * sh.n2 != uint64_t (sh.nsub) * sh.freq_res || sh.seg * sh.nsub != sh.n2
      || sh.npol < 1 || sh.npol > 2 || in.fb_nsub)
    return cudaErrorInvalidValue;
  switch (sh.n1)
  {
    case 2: return run_during_n1<2> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 4: return run_during_n1<4> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 8: return run_during_n1<8> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 16: return run_during_n1<16> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 32: return run_during_n1<32> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 64: return run_during_big<64> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 128:
      return run_during_big<128> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 256:
      return run_during_big<256> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    case 512:
      return run_during_big<512> (sh, tb, in, part0, nbatch, scratch, mode, fv, vv, st, clk);
    default: return cudaErrorInvalidValue;
  }
}

} // namespace b200
