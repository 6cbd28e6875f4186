// ifb.cu -- inverse filterbank kernels (InverseFilterbankEngineCPU.C)

#include "fb_warp.cuh"
#include "group_fft.cuh"
#include "rows32.cuh"

namespace b200 {

namespace {

// --------------------------------------------------------------------------
// inverse filterbank (InverseFilterbankEngineCPU.C:309-779 restructured)
// --------------------------------------------------------------------------

// The kept bins of one (channel, pol) spectrum (s, padded layout) to the
// output channels' spectra, by the TF threads of the transform (tid).
template <int LIN, int TF>
__device__ __forceinline__ void stitch_out (const float2* s, const IfbShape& sh,
                                            const IfbTables& tb, float2* __restrict__ scratch,
                                            unsigned b, unsigned c, unsigned p, unsigned tid)
{
  const int4 m = __ldg (tb.map + c);
  const unsigned keep2 = sh.keep / 2;
  const unsigned skip2 = (LIN - sh.keep) / 2;
  const unsigned src_neg = sh.dual_sideband ? LIN - keep2 : skip2;
  const unsigned src_pos = sh.dual_sideband ? 0 : skip2 + keep2;
  if (keep2 % sh.n1 == 0)
  {
    // n1 divides keep/2, so every half starts on a multiple of n1 and its
    // bins fill per_row consecutive columns of each four-step row: threads
    // walk them row by row, consecutive threads writing consecutive columns.
    const unsigned per_row = keep2 / sh.n1;
    const bool pow2 = (per_row & (per_row - 1)) == 0;
    const unsigned lg = __ffs (per_row) - 1;
    for (int h = 0; h < 2; h++)
    {
      const int o = h ? m.z : m.x;
      const int offz = h ? m.w : m.y;
      const unsigned off = unsigned (offz & (IFB_ZERO - 1));
      const unsigned src0 = h ? src_pos : src_neg;
      float2* dst = scratch + ((uint64_t (b) * sh.nout + o) * sh.npol + p) * sh.lout + off / sh.n1;
      // where whole rows fill the group, a lane keeps its column and steps by
      // whole rows: a third of the general loop's instructions per bin (758
      // against 661 us for the stitch of 256 x 1024 points)
      if (pow2 && per_row <= unsigned (TF) && !(offz & IFB_ZERO) && !tb.response && !tb.spectral)
      {
        const unsigned a0 = tid >> lg, q = tid & (per_row - 1), da = TF >> lg;
        unsigned i = src0 + q * sh.n1 + a0;
        unsigned k = a0 * sh.n2 + q;
#pragma unroll 4
        for (unsigned a = a0; a < sh.n1; a += da, i += da, k += da * sh.n2) dst[k] = s[spad (i)];
        continue;
      }
      for (unsigned r = tid; r < keep2; r += TF)
      {
        const unsigned a = pow2 ? r >> lg : r / per_row;
        const unsigned q = r - a * per_row;
        const unsigned j = q * sh.n1 + a;
        float2 y = (offz & IFB_ZERO) ? make_float2 (0.f, 0.f) : s[spad (src0 + j)];
        if (tb.response)
        {
          const float2 f = __ldg (tb.response + uint64_t (o) * sh.lout + off + j);
          y = make_float2 (__fsub_rn (__fmul_rn (f.x, y.x), __fmul_rn (f.y, y.y)),
                           __fadd_rn (__fmul_rn (f.y, y.x), __fmul_rn (f.x, y.y)));
        }
        if (tb.spectral)
        {
          const float w = __ldg (tb.spectral + off + j);
          y = make_float2 (__fmul_rn (y.x, w), __fmul_rn (y.y, w));
        }
        dst[uint64_t (a) * sh.n2 + q] = y;
      }
    }
    return;
  }
  for (unsigned i = tid; i < sh.keep; i += TF)
  {
    const bool neg = i < keep2;
    const unsigned j = neg ? i : i - keep2;
    const int o = neg ? m.x : m.z;
    const int off = neg ? m.y : m.w;
    const unsigned k = unsigned (off & (IFB_ZERO - 1)) + j;
    float2 y = (off & IFB_ZERO) ? make_float2 (0.f, 0.f) : s[spad ((neg ? src_neg : src_pos) + j)];
    if (tb.response)
    {
      // Response::operate: (f_r d_r - f_i d_i, f_i d_r + f_r d_i)
      const float2 f = __ldg (tb.response + uint64_t (o) * sh.lout + k);
      y = make_float2 (__fsub_rn (__fmul_rn (f.x, y.x), __fmul_rn (f.y, y.y)),
                       __fadd_rn (__fmul_rn (f.y, y.x), __fmul_rn (f.x, y.y)));
    }
    if (tb.spectral)
    {
      const float w = __ldg (tb.spectral + k);
      y = make_float2 (__fmul_rn (y.x, w), __fmul_rn (y.y, w));
    }
    float2* dst = scratch + ((uint64_t (b) * sh.nout + o) * sh.npol + p) * sh.lout;
    dst[uint64_t (k % sh.n1) * sh.n2 + k / sh.n1] = y;
  }
}

// A CTA of IFB_THREADS threads transforms F = 8192/LIN (channel, pol) slots of
// one part: CG = F/npol consecutive fine channels, both pols.  The input tile
// is read so that consecutive threads touch consecutive bytes (for TFPD input
// the slots of one time sample are contiguous; for FPT input the samples of
// one slot are), unpacked and windowed (Apodization::operate) into shared
// memory; each group of LIN/16 threads runs the forward FFT of its slot; then
// the kept bins of both halves -- stitch_one's placement, precomputed per
// channel on the host -- times the response and the spectral window go to the
// output channel's spectrum in four-step order (bin k at row k mod n1, column
// k div n1) for the row kernel.
constexpr int IFB_THREADS = 512;

template <int LIN, int KIND>
__global__ void __launch_bounds__ (IFB_THREADS)
k_ifb_stitch (const InputView in, const IfbShape sh, const IfbTables tb, const uint64_t part0,
              float2* __restrict__ scratch)
{
  constexpr int TF = stockham_threads (LIN);     // threads per transform
  constexpr int F = IFB_THREADS / TF;             // slots per CTA
  // slot stride: the padded transform plus 32 bytes, so that the slots of one
  // time sample written together fall on different banks
  constexpr int SP = spad_size (LIN) + 4;
  constexpr int TABN = pass_tables_size (LIN);
  extern __shared__ float2 s_ifb[];               // [F][SP], then the pass tables
  float2* s_tab = s_ifb + F * SP;
  __shared__ float s_lut[256];
  const unsigned npol = sh.npol;
  const unsigned cg = F / npol;                   // channels per CTA
  const unsigned c0 = blockIdx.x * cg;
  const unsigned b = blockIdx.y;
  load_lut (in, tb.lut, s_lut);
  for (int i = threadIdx.x; i < TABN; i += IFB_THREADS) s_tab[i] = __ldg (tb.ptab_lin + i);
  __syncthreads ();
  const uint64_t t0 = (part0 + b) * sh.in_step;
  // all PER loads of a thread are issued before any is used
  constexpr int PER = F * LIN / IFB_THREADS;
  const unsigned nslot = min (unsigned (F), (sh.nin - c0) * npol);   // live slots
  const uint64_t row = uint64_t (sh.nin) * npol;                       // TFPD values per sample
  uint32_t word[PER];
  float2 fv[KIND == IN_FLOAT ? PER : 1];
#pragma unroll
  for (int k = 0; k < PER; k++)
  {
    const unsigned e = threadIdx.x + k * IFB_THREADS;
    if constexpr (KIND == IN_FLOAT)
    {
      const unsigned slot = e / LIN, t = e % LIN;
      fv[k] = slot < nslot ? __ldg (static_cast<const float2*> (in.main)
                                    + (uint64_t (c0) * npol + slot) * in.main_span + t0 + t)
                           : make_float2 (0.f, 0.f);
    }
    else
    {
      const unsigned slot = e % F, t = e / F;
      const uint64_t idx = (t0 + t) * row + uint64_t (c0) * npol + slot;
      if constexpr (KIND == IN_INT16)
        word[k] = slot < nslot ? __ldg (static_cast<const uint32_t*> (in.main) + idx) : 0u;
      else
        word[k] = slot < nslot ? __ldg (static_cast<const unsigned short*> (in.main) + idx) : 0u;
    }
  }
#pragma unroll
  for (int k = 0; k < PER; k++)
  {
    const unsigned e = threadIdx.x + k * IFB_THREADS;
    unsigned slot, t;
    float2 x;
    if constexpr (KIND == IN_FLOAT)
    {
      slot = e / LIN;
      t = e % LIN;
      x = fv[k];
    }
    else
    {
      slot = e % F;
      t = e / F;
      if constexpr (KIND == IN_INT16)
      {
        short re = short (word[k] & 0xffff), im = short (word[k] >> 16);
        if (in.offset_binary)
        {
          re = short (re ^ 0x8000);
          im = short (im ^ 0x8000);
        }
        // SixteenBitUnpacker.C:69: float(x) + 0.5
        x = make_float2 (__fadd_rn (float (re), 0.5f), __fadd_rn (float (im), 0.5f));
      }
      else
        x = make_float2 (s_lut[word[k] & 0xff], s_lut[word[k] >> 8]);
      if (slot >= nslot) x = make_float2 (0.f, 0.f);
    }
    if (tb.temporal)
    {
      const float w = __ldg (tb.temporal + t);
      x = make_float2 (__fmul_rn (x.x, w), __fmul_rn (x.y, w));
    }
    s_ifb[slot * SP + spad (t)] = x;
  }
  __syncthreads ();
  const unsigned group = threadIdx.x / TF, tid = threadIdx.x % TF;
  float2* s = s_ifb + group * SP;
  {
    float2 v[LIN / TF];
    group_fft_pass<LIN, TF, -1, 0> (s, v, s_tab, tid);
  }
  const unsigned c = c0 + group / npol, p = group % npol;
  if (c < sh.nin) stitch_out<LIN, TF> (s, sh, tb, scratch, b, c, p, tid);
}

// The same for LIN = 256 .. 1024 with 32 points per thread (FbWarp's split
// LIN = 32 x M: one exchange, warp barriers only), where ifb_stitch_by_warps
// chooses it.  A block takes
// 8 * (32 / M) slots; TFPD samples are loaded in address order (all slots of a
// time sample together) and handed over as raw words in the slots' own
// regions, whose stride of 4 mod 32 words keeps both sides free of bank
// conflicts; FPT samples are loaded by the slot's own lanes.  16 points per
// thread in three block-wide passes moved 80 bytes per point through shared
// memory, this 48: 790 us before, 758 us with it for 256 channels of
// 1024 points.
template <int LIN, int KIND>
__global__ void __launch_bounds__ (FBW_WARPS * 32, 2)
k_ifb_stitch_warp (const InputView in, const IfbShape sh, const IfbTables tb, const uint64_t part0,
                   float2* __restrict__ scratch)
{
  using FW = FbWarp<LIN>;
  constexpr int M = FW::M;
  constexpr int T = FBW_WARPS * 32;
  constexpr unsigned F = FW::NB;                   // slots per block
  static_assert (spad_size (LIN) <= FW::RS, "the spectrum fits its region");
  extern __shared__ __align__ (16) float2 s_ifw[];
  float2* tw = s_ifw + F * FW::RS;                 // w_LIN^(q t) at [q * M + t]
  __shared__ float s_lut[KIND == IN_INT8 ? 256 : 1];
  const unsigned npol = sh.npol;
  const unsigned c0 = blockIdx.x * (F / npol);
  const unsigned b = blockIdx.y;
  if constexpr (KIND == IN_INT8) load_lut (in, tb.lut, s_lut);
  for (int i = threadIdx.x; i < LIN; i += T)
  {
    // w_LIN^m is w_1024^(m 1024 / LIN)
    const int m = (i / M) * (i % M) % LIN;
    tw[i] = __ldg (tb.tw1024 + m * (1024 / LIN));
  }
  const uint64_t t0 = (part0 + b) * sh.in_step;
  const unsigned nslot = min (F, (sh.nin - c0) * npol);                // live slots
  const int t = threadIdx.x % M;
  const unsigned slot = threadIdx.x / M;
  float2* s = s_ifw + slot * FW::RS;
  CP v[32];
  if constexpr (KIND == IN_FLOAT)
  {
#pragma unroll
    for (int r = 0; r < 32; r++)
      v[r].z = slot < nslot ? __ldg (static_cast<const float2*> (in.main)
                                     + (uint64_t (c0) * npol + slot) * in.main_span + t0 + t + M * r)
                            : make_float2 (0.f, 0.f);
    __syncthreads ();                  // the twiddles are there
  }
  else
  {
    const uint64_t row = uint64_t (sh.nin) * npol;                     // TFPD values per sample
    uint32_t word[32];
#pragma unroll
    for (int k = 0; k < 32; k++)
    {
      const unsigned e = threadIdx.x + k * T, sl = e % F, tt = e / F;
      const uint64_t idx = (t0 + tt) * row + uint64_t (c0) * npol + sl;
      if constexpr (KIND == IN_INT16)
        word[k] = sl < nslot ? __ldg (static_cast<const uint32_t*> (in.main) + idx) : 0u;
      else
        word[k] = sl < nslot ? __ldg (static_cast<const unsigned short*> (in.main) + idx) : 0u;
    }
    uint32_t* raw = reinterpret_cast<uint32_t*> (s_ifw);
#pragma unroll
    for (int k = 0; k < 32; k++)
    {
      const unsigned e = threadIdx.x + k * T;
      raw[(e % F) * (2 * FW::RS) + e / F] = word[k];
    }
    __syncthreads ();
#pragma unroll
    for (int r = 0; r < 32; r++)
    {
      const uint32_t w = raw[slot * (2 * FW::RS) + t + M * r];
      float2 x;
      if constexpr (KIND == IN_INT16)
      {
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
        x = make_float2 (s_lut[w & 0xff], s_lut[w >> 8]);
      v[r].z = slot < nslot ? x : make_float2 (0.f, 0.f);
    }
  }
  if (tb.temporal)
  {
#pragma unroll
    for (int r = 0; r < 32; r++)
    {
      const float w = __ldg (tb.temporal + t + M * r);
      v[r].z = make_float2 (__fmul_rn (v[r].z.x, w), __fmul_rn (v[r].z.y, w));
    }
  }
  dft::run<32, -1> (v);
  __syncwarp ();                       // the raw words of the warp's slots have been read
#pragma unroll
  for (int q = 0; q < 32; q++) s[q * FW::LD + t] = q ? cmul (v[q].z, tw[q * M + t]) : v[q].z;
  __syncwarp ();
#pragma unroll
  for (int i = 0; i < FW::G; i++)
#pragma unroll
    for (int j = 0; j < M / 2; j++)
    {
      const float4 x = *reinterpret_cast<const float4*> (s + (t + M * i) * FW::LD + 2 * j);
      v[i * M + 2 * j].z = make_float2 (x.x, x.y);
      v[i * M + 2 * j + 1].z = make_float2 (x.z, x.w);
    }
  __syncwarp ();
#pragma unroll
  for (int i = 0; i < FW::G; i++)
  {
    dft::run<M, -1> (v + i * M);
#pragma unroll
    for (int p = 0; p < M; p++) s[spad (t + M * i + 32 * p)] = v[i * M + p].z;
  }
  __syncwarp ();
  if (slot < nslot)
    stitch_out<LIN, M> (s, sh, tb, scratch, b, c0 + slot / npol, slot % npol, t);
}

// Inverse column DFTs of the lout-point transforms (after the row kernel):
// conjugate four-step twiddle, n1-point inverse DFT in registers (n1 may
// carry a factor 3), output discard, voltages out.  Pols one after another.
template <int N1>
__global__ void __launch_bounds__ (128)
k_ifb_cols (const float2* __restrict__ scratch, const IfbShape sh, const float2* __restrict__ tw4,
            const uint64_t part0, const VoltView vv)
{
  const unsigned i2 = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned b = blockIdx.y;
  const unsigned o = blockIdx.z;
  const uint64_t N = uint64_t (N1) * sh.n2;
  const uint64_t tbase = (part0 + b) * sh.out_step;
  for (unsigned p = 0; p < sh.npol; p++)
  {
    const float2* src = scratch + ((uint64_t (b) * sh.nout + o) * sh.npol + p) * N + i2;
    float2 v[N1];
#pragma unroll
    for (int k = 0; k < N1; k++) v[k] = src[uint64_t (k) * sh.n2];
#pragma unroll
    for (int k = 1; k < N1; k++) v[k] = cmulc (v[k], __ldg (tw4 + uint64_t (k) * sh.n2 + i2));
    RegDFTm<N1, +1>::run (v);
    float2* dst = vv.out + (uint64_t (o) * sh.npol + p) * vv.span + tbase;
#pragma unroll
    for (int k = 0; k < N1; k++)
    {
      const uint64_t tl = uint64_t (k) * sh.n2 + i2;
      if (tl >= sh.out_discard_pos && tl < sh.out_discard_pos + sh.out_step)
        dst[tl - sh.out_discard_pos] = v[k];
    }
  }
}

template <int LIN, int KIND>
void launch_ifb_stitch (const IfbShape& sh, const IfbTables& tb, const InputView& in,
                        uint64_t part0, unsigned nbatch, float2* scratch, cudaStream_t st)
{
  constexpr int F = IFB_THREADS / stockham_threads (LIN);
  const size_t smem = (size_t (F) * (spad_size (LIN) + 4) + pass_tables_size (LIN)) * sizeof (float2);
  auto kern = k_ifb_stitch<LIN, KIND>;
  cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
  const unsigned cg = F / sh.npol;
  kern<<<dim3 ((sh.nin + cg - 1) / cg, nbatch), IFB_THREADS, smem, st>>> (in, sh, tb, part0,
                                                                         scratch);
}

template <int LIN, int KIND>
void launch_ifb_stitch_warp (const IfbShape& sh, const IfbTables& tb, const InputView& in,
                             uint64_t part0, unsigned nbatch, float2* scratch, cudaStream_t st)
{
  using FW = FbWarp<LIN>;
  auto kern = k_ifb_stitch_warp<LIN, KIND>;
  cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int (FW::SMEM));
  const unsigned cg = FW::NB / sh.npol;
  kern<<<dim3 ((sh.nin + cg - 1) / cg, nbatch), FBW_WARPS * 32, FW::SMEM, st>>> (in, sh, tb, part0,
                                                                                scratch);
}

// Whether the transforms of lin points run 32 points per thread.  That spends
// less on the transform and shared memory, but leaves half the threads to place
// the bins: a response or a spectral window, loaded bin by bin, then costs more
// than the transform gains, except for float samples, and so do 128-point
// transforms, which make the most slots.  Calls of 64 M samples, 16 points per
// thread / 32 (us): 1024 x 256 int16 1322 / 1218, with a response 1478 / 1433;
// 1024 x 64 int16, one polarisation 634 / 626, with a response 656 / 683;
// 256 x 128 int16 640 / 632, with a response 648 / 712, int8 1276 / 1307;
// 128 x 256 float 655 / 683.
bool ifb_stitch_by_warps (unsigned lin, int kind, bool windows)
{
  if (lin == 256) return kind != IN_INT8 && !windows;
  return (lin == 512 || lin == 1024) && (kind == IN_FLOAT || !windows);
}

template <int LIN>
void launch_ifb_stitch_k (const IfbShape& sh, const IfbTables& tb, const InputView& in,
                          uint64_t part0, unsigned nbatch, float2* scratch, cudaStream_t st)
{
  if constexpr (LIN >= 256 && LIN <= 1024)
    if (ifb_stitch_by_warps (LIN, in.kind, tb.response || tb.spectral))
    {
      if (in.kind == IN_INT16)
        launch_ifb_stitch_warp<LIN, IN_INT16> (sh, tb, in, part0, nbatch, scratch, st);
      else if (in.kind == IN_FLOAT)
        launch_ifb_stitch_warp<LIN, IN_FLOAT> (sh, tb, in, part0, nbatch, scratch, st);
      else if constexpr (LIN >= 512)
        launch_ifb_stitch_warp<LIN, IN_INT8> (sh, tb, in, part0, nbatch, scratch, st);
      return;
    }
  if (in.kind == IN_INT8)
    launch_ifb_stitch<LIN, IN_INT8> (sh, tb, in, part0, nbatch, scratch, st);
  else if (in.kind == IN_INT16)
    launch_ifb_stitch<LIN, IN_INT16> (sh, tb, in, part0, nbatch, scratch, st);
  else
    launch_ifb_stitch<LIN, IN_FLOAT> (sh, tb, in, part0, nbatch, scratch, st);
}

template <int N1>
void launch_ifb_cols (const IfbShape& sh, const IfbTables& tb, uint64_t part0, unsigned nbatch,
                      const float2* scratch, const VoltView& vv, cudaStream_t st)
{
  k_ifb_cols<N1><<<dim3 (sh.n2 / 128, nbatch, sh.nout), 128, 0, st>>> (scratch, sh, tb.tw4, part0,
                                                                       vv);
}

template <int N2>
void launch_rows_inv (unsigned nrows, float2* scratch, const IfbTables& tb, unsigned n1,
                      unsigned npol, cudaStream_t st)
{
  const unsigned grid = std::min<unsigned> (nrows, rows32_ctas_per_sm<N2> () * unsigned (tb.nsm));
  k_rows32<N2, false><<<grid, Row32<N2>::T, rows32_smem_bytes<N2> (), st>>> (
      scratch, nullptr, n1, 1, npol, nrows, nrows / n1);
}

} // namespace

bool ifb_supported_lin (unsigned lin)
{
  return lin == 64 || lin == 128 || lin == 256 || lin == 512 || lin == 1024 || lin == 2048 ||
         lin == 4096;
}

cudaError_t inverse_filterbank_kernel_setup ()
{
  static std::atomic<unsigned> done {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess) return e;
  const unsigned bit = dev < 32 ? 1u << dev : 0u;    // devices past 32: set every time
  if (bit && (done.load () & bit)) return cudaSuccess;
  e = set_rows_smem<8192, false> ();
  if (e == cudaSuccess) e = set_rows_smem<4096, false> ();
  if (e == cudaSuccess) done.fetch_or (bit);
  return e;
}

cudaError_t launch_inverse_filterbank (const IfbShape& sh, const IfbTables& tb,
                                       const InputView& in, uint64_t part0, unsigned nbatch,
                                       float2* scratch, const VoltView& vv, cudaStream_t st,
                                       const KernelClock* clk)
{
  if (nbatch == 0) return cudaSuccess;
  if (sh.n2 != 8192 && sh.n2 != 4096) return cudaErrorInvalidValue;
  {
    const cudaError_t e = inverse_filterbank_kernel_setup ();
    if (e != cudaSuccess) return e;
  }
  {
    ClockScope cs (clk, KK_FWD_COLS, st);
    switch (sh.lin)
    {
      case 64: launch_ifb_stitch_k<64> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 128: launch_ifb_stitch_k<128> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 256: launch_ifb_stitch_k<256> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 512: launch_ifb_stitch_k<512> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 1024: launch_ifb_stitch_k<1024> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 2048: launch_ifb_stitch_k<2048> (sh, tb, in, part0, nbatch, scratch, st); break;
      case 4096: launch_ifb_stitch_k<4096> (sh, tb, in, part0, nbatch, scratch, st); break;
      default: return cudaErrorInvalidValue;
    }
  }
  const unsigned nrows = sh.n1 * nbatch * sh.nout * sh.npol;
  {
    ClockScope cs (clk, KK_ROWS, st);
    if (sh.n2 == 8192)
      launch_rows_inv<8192> (nrows, scratch, tb, sh.n1, sh.npol, st);
    else
      launch_rows_inv<4096> (nrows, scratch, tb, sh.n1, sh.npol, st);
  }
  ClockScope cs (clk, KK_INV_COLS, st);
  switch (sh.n1)
  {
    case 2: launch_ifb_cols<2> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 3: launch_ifb_cols<3> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 4: launch_ifb_cols<4> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 6: launch_ifb_cols<6> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 8: launch_ifb_cols<8> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 12: launch_ifb_cols<12> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 16: launch_ifb_cols<16> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 24: launch_ifb_cols<24> (sh, tb, part0, nbatch, scratch, vv, st); break;
    case 32: launch_ifb_cols<32> (sh, tb, part0, nbatch, scratch, vv, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError ();
}

} // namespace b200
