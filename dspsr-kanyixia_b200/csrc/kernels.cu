// kernels.cu -- response construction and the standalone engines: filterbank,
// SpectralKurtosis, unpackers, detection, fold (sm_100a)

#include "device_common.cuh"
#include "fb_warp.cuh"
#include "fwd_cols_pair.cuh"
#include "group_fft.cuh"

namespace b200 {

std::atomic<uint64_t> g_launches {0};

namespace {

// --------------------------------------------------------------------------
// response construction
// --------------------------------------------------------------------------

// Dedispersion::build_compute (Dedispersion.C:166-186) on the grid of the
// restated PlasmaResponse::build: channel ichan centred at chan_freq, bin ipt
// at freq = ipt*binwidth - chanwidth/2 (natural order).  FFT-order index k
// maps to ipt = k + N/2 (mod N) when the halves are swapped
// (Response::doswap, Response.C:998-1050).  Written in four-step order
// H[c][k1][k2] for k = k1 + n1*k2.
__global__ void k_build_chirp (float2* __restrict__ H, const double* __restrict__ chan_freq,
                               const double* __restrict__ coeff, const double* __restrict__ frac_us,
                               const unsigned nfft, const unsigned n1, const unsigned n2,
                               const double binwidth, const double half_chanwidth,
                               const int swap_halves, const int chirp_mode, const float scale)
{
  const uint64_t idx = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (idx >= nfft) return;
  const unsigned k1 = unsigned (idx / n2), k2 = unsigned (idx % n2);
  const unsigned k = k1 + n1 * k2;
  const unsigned ipt = swap_halves ? (k + nfft / 2) % nfft : k;
  const double cf = chan_freq[c];
  const double freq = __dsub_rn (__dmul_rn (double (ipt), binwidth), half_chanwidth);
  const double num = __dmul_rn (coeff[c], __dmul_rn (freq, freq));
  double phase = __ddiv_rn (num, __dadd_rn (cf, freq));
  if (frac_us)
  {
    // Dedispersion::build_compute (Dedispersion.C:176-179): the phase of the
    // channel's fractional-sample inter-channel delay
    const double minus_two_pi = -6.283185307179586476925286766559;
    phase = __dadd_rn (phase, __dmul_rn (__dmul_rn (minus_two_pi, freq), frac_us[c]));
  }
  float re, im;
  if (chirp_mode == 0)
  {
    // Dedispersion.C:104-111: phases stored as float, then polar(1.0f, phase)
    const float ph = __double2float_rn (phase);
    sincosf (ph, &im, &re);
  }
  else
  {
    const double two_pi = 6.283185307179586476925286766559;
    const double red = __dsub_rn (phase, __dmul_rn (two_pi, rint (__ddiv_rn (phase, two_pi))));
    double s, co;
    sincos (red, &s, &co);
    re = __double2float_rn (co);
    im = __double2float_rn (s);
  }
  H[uint64_t (c) * nfft + idx] = make_float2 (__fmul_rn (re, scale), __fmul_rn (im, scale));
}

__global__ void k_permute (float2* __restrict__ dst, const float2* __restrict__ src,
                           const unsigned n1, const unsigned n2, const int inverse)
{
  const uint64_t N = uint64_t (n1) * n2;
  const uint64_t idx = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (idx >= N) return;
  const unsigned k1 = unsigned (idx / n2), k2 = unsigned (idx % n2);
  const uint64_t k = k1 + uint64_t (n1) * k2;
  if (inverse)
    dst[c * N + k] = src[c * N + idx];
  else
    dst[c * N + idx] = src[c * N + k];
}

// --------------------------------------------------------------------------
// standalone engines
// --------------------------------------------------------------------------

// FFT filterbank without convolution (Filterbank with freq_res = 1,
// FilterbankEngineCPU.C:379-535): every block of NSUB input samples becomes one
// sample in each of NSUB output channels, channel k = FFT bin k scaled by the
// normaliser 1/sqrt(NSUB) (Filterbank.C:171-180).  The unpack is fused into
// the load; one thread transforms one block of one polarisation in registers.
template <int NSUB, int KIND>
__global__ void __launch_bounds__ (128)
k_filterbank (const InputView in, const float* __restrict__ lut, const uint64_t nblk,
              const float scale, float2* __restrict__ out, const uint64_t out_span)
{
  __shared__ float s_lut[256];
  load_lut (in, lut, s_lut);
  __syncthreads ();
  const uint64_t blk = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned p = blockIdx.y;
  const unsigned cin = blockIdx.z;
  if (blk >= nblk) return;
  float2 v[NSUB];
#pragma unroll
  for (int k = 0; k < NSUB; k++)
    v[k] = fetch<KIND> (in, s_lut, cin, p, blk * NSUB + k);
  RegDFT<NSUB, -1>::run (v);
  float2* o = out + (uint64_t (cin) * NSUB * in.npol + p) * out_span + blk;
#pragma unroll
  for (int k = 0; k < NSUB; k++)
    o[uint64_t (k) * in.npol * out_span] = make_float2 (__fmul_rn (scale, v[k].x),
                                                         __fmul_rn (scale, v[k].y));
}

// The same filterbank for NSUB = 2048 and 4096 with the transforms in shared
// memory: a CTA of FB_THREADS threads takes F = 8192/NSUB (block, pol) slots of
// one input channel, reads their samples in address order (coalesced), runs
// one NSUB-point FFT per group of NSUB/16 threads (per-pass twiddle tables in
// shared memory), and writes the bins channel by channel, consecutive threads
// on consecutive output samples.
constexpr int FB_THREADS = 512;

template <int NSUB, int KIND>
__global__ void __launch_bounds__ (FB_THREADS)
k_filterbank_smem (const InputView in, const float* __restrict__ lut, const float2* __restrict__ ptab,
                   const uint64_t nblk, const float scale, float2* __restrict__ out,
                   const uint64_t out_span)
{
  constexpr int TF = stockham_threads (NSUB);
  constexpr int F = FB_THREADS / TF;
  // odd slot stride (in float2): the output loop reads one bin of consecutive
  // slots, which then fall on different banks
  constexpr int SP = spad_size (NSUB) + 1;
  constexpr int TABN = pass_tables_size (NSUB);
  extern __shared__ float2 s_fb[];                 // [F][SP], then the pass tables
  float2* s_tab = s_fb + F * SP;
  __shared__ float s_lut[256];
  const unsigned npol = in.npol;
  const unsigned bpc = F / npol;                    // blocks per CTA
  const uint64_t blk0 = uint64_t (blockIdx.x) * bpc;
  const unsigned cin = blockIdx.y;
  const unsigned nb = unsigned (min (uint64_t (bpc), nblk - blk0));
  load_lut (in, lut, s_lut);
  for (int i = threadIdx.x; i < TABN; i += FB_THREADS) s_tab[i] = __ldg (ptab + i);
  __syncthreads ();
  const uint64_t t0 = blk0 * NSUB;
  // element e in address order: TFPD (t, pol) pairs, FPT (pol, t); all PER
  // loads of a thread are issued before any is used
  constexpr int PER = F * NSUB / FB_THREADS;
  constexpr unsigned HALF = F * NSUB / 2;          // samples per pol when npol == 2
  const bool two = npol == 2;
  const uint64_t rowv = uint64_t (in.nchan) * npol;  // TFPD values per time sample
  uint32_t word[PER];
  float2 fv[KIND == IN_FLOAT ? PER : 1];
#pragma unroll
  for (int k = 0; k < PER; k++)
  {
    const unsigned e = threadIdx.x + k * FB_THREADS;
    if constexpr (KIND == IN_FLOAT)
    {
      const unsigned p = two ? e / HALF : 0, t = two ? e % HALF : e;
      fv[k] = t / NSUB < nb ? __ldg (static_cast<const float2*> (in.main)
                                     + (uint64_t (cin) * npol + p) * in.main_span + t0 + t)
                            : make_float2 (0.f, 0.f);
    }
    else
    {
      const unsigned p = two ? (e & 1) : 0, t = two ? e >> 1 : e;
      const uint64_t idx = (t0 + t) * rowv + uint64_t (cin) * npol + p;
      if constexpr (KIND == IN_INT16)
        word[k] = t / NSUB < nb ? __ldg (static_cast<const uint32_t*> (in.main) + idx) : 0u;
      else
        word[k] = t / NSUB < nb ? __ldg (static_cast<const unsigned short*> (in.main) + idx) : 0u;
    }
  }
#pragma unroll
  for (int k = 0; k < PER; k++)
  {
    const unsigned e = threadIdx.x + k * FB_THREADS;
    unsigned p, t;
    float2 x;
    if constexpr (KIND == IN_FLOAT)
    {
      p = two ? e / HALF : 0;
      t = two ? e % HALF : e;
      x = fv[k];
    }
    else
    {
      p = two ? (e & 1) : 0;
      t = two ? e >> 1 : e;
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
    }
    const unsigned blk = t / NSUB, i = t % NSUB;
    if (blk >= nb) x = make_float2 (0.f, 0.f);
    s_fb[(blk * npol + p) * SP + spad (i)] = x;
  }
  __syncthreads ();
  const unsigned group = threadIdx.x / TF, tid = threadIdx.x % TF;
  {
    float2 v[NSUB / TF];
    group_fft_pass<NSUB, TF, -1, 0> (s_fb + group * SP, v, s_tab, tid);
  }
  // bins out: channel cin*NSUB + k of pol p, sample blk0 + blk
  for (unsigned e = threadIdx.x; e < unsigned (F * NSUB); e += FB_THREADS)
  {
    const unsigned blk = e % bpc, rest = e / bpc;
    const unsigned p = rest % npol, k = rest / npol;
    if (blk >= nb || k >= NSUB) continue;
    const float2 y = s_fb[(blk * npol + p) * SP + spad (k)];
    out[((uint64_t (cin) * NSUB + k) * npol + p) * out_span + blk0 + blk] =
        make_float2 (__fmul_rn (scale, y.x), __fmul_rn (scale, y.y));
  }
}

// SpectralKurtosis::transformation for one resolution with noverlap = 1:
// compute (SpectralKurtosis.C:674-798), detect_skfb (:1105-1222) and mask
// (:1465-1566).  A CTA takes up to U consecutive M-sample blocks of one
// channel:
//
//   1. all threads stream the blocks in (16-byte loads, both pols in flight
//      together), square-law detect them in float as the reference does and
//      keep sqld per (block, pol) in shared memory; out of place the voltages
//      are written through to the output at the same time;
//   2. warp 0 forms the reference's two sequential double sums per (block,
//      pol) -- S1 of sqld, S2 of sqld*sqld -- one lane per sum, 4U lanes in
//      all, so that each conversion to double serves 4U values.  The
//      additions run in the reference's order: the sums (and hence the mask)
//      equal the CPU's bit for bit.  Many CTAs per SM keep the loads of some
//      in flight while others add;
//   3. the SK estimator of each block is tested and zapped blocks of the
//      output are overwritten with zeros (in place, only they are written).
//
// Uncounted samples (sqld == 0 with zero_is_valid unset) add +0.0, which
// leaves a sum of non-negative terms unchanged exactly; they are counted by a
// shared atomic as they are met.  Shared memory holds U * npol columns of
// Ms floats, Ms = M rounded up to a multiple of 4 plus 4 (so that the
// columns read together fall on different banks).
// Bound by HBM (16 B per sample) where M is short and by the chains of double
// additions where it is long.  With a load behind each store, 128 threads and
// two blocks per CTA 512 channels x 131072 samples took 459 us at M = 1024 and
// 536 us at M = 256; now 376 and 329 us (6.5 TB/s).  More threads or blocks per
// CTA (eight blocks, 512 threads) took 440 to 505 us at M = 1024, streaming
// hints on the loads and stores 388.
constexpr int SK_THREADS = 256;
constexpr size_t SK_TILE = 40u << 10;           // five CTAs per SM
constexpr int SK_BATCH = 4;

__host__ __device__ inline unsigned sk_column (unsigned M) { return ((M + 3) & ~3u) + 4; }

template <int U>
__global__ void __launch_bounds__ (SK_THREADS, 5)
k_sk (const float2* __restrict__ in, const uint64_t in_span, float2* out, const uint64_t out_span,
      const uint64_t npart, const unsigned nchan, const unsigned npol, const unsigned M,
      const int zero_is_valid, const unsigned Nd, const float lower,
      const float upper, float* __restrict__ sums, unsigned* __restrict__ counts,
      uint8_t* __restrict__ mask, unsigned long long* __restrict__ nzap)
{
  extern __shared__ __align__ (16) float s_sqld[];   // [unit][pol][Ms]
  __shared__ double s_sum[U][2][2];
  __shared__ unsigned s_zero[U];
  __shared__ int s_zap[U];
  const uint64_t part0 = uint64_t (blockIdx.x) * U;
  const unsigned c = blockIdx.y;
  const unsigned nu = unsigned (min (uint64_t (U), npart - part0));
  const unsigned Ms = sk_column (M);
  const unsigned n4 = M / 2;                      // float4 (two samples) per (block, pol)
  // out == nullptr: statistics only (SpectralKurtosis::compute), nothing written back
  const bool through = out && !(out == in && out_span == in_span);
  const bool two = npol == 2;
  if (threadIdx.x < U) s_zero[threadIdx.x] = 0;
  // both pols of the CTA's blocks are contiguous runs of nu*M samples
  const float4* src0 = reinterpret_cast<const float4*> (in + uint64_t (c) * npol * in_span
                                                        + part0 * M);
  const float4* src1 = src0 + (two ? in_span / 2 : 0);
  float4* dst0 = reinterpret_cast<float4*> (out + uint64_t (c) * npol * out_span + part0 * M);
  float4* dst1 = dst0 + (two ? out_span / 2 : 0);
  __syncthreads ();
  const unsigned total = nu * n4;
  // SK_BATCH loads per polarisation are issued before any is used: the stores
  // may alias the loads, and the compiler would keep each load behind the
  // store before it
  for (unsigned f0 = threadIdx.x; f0 < total; f0 += SK_BATCH * SK_THREADS)
  {
    float4 a[SK_BATCH], b[SK_BATCH];
#pragma unroll
    for (int k = 0; k < SK_BATCH; k++)
    {
      const unsigned f = f0 + k * SK_THREADS;
      a[k] = b[k] = make_float4 (1.f, 1.f, 1.f, 1.f);
      if (f < total)
      {
        a[k] = src0[f];
        if (two) b[k] = src1[f];
      }
    }
#pragma unroll
    for (int k = 0; k < SK_BATCH; k++)
    {
      const unsigned f = f0 + k * SK_THREADS;
      if (f >= total) break;
      if (through)
      {
        dst0[f] = a[k];
        if (two) dst1[f] = b[k];
      }
      const unsigned u = U == 1 || f < n4 ? 0 : f / n4, i = f - u * n4;
      const float a0 = __fadd_rn (__fmul_rn (a[k].x, a[k].x), __fmul_rn (a[k].y, a[k].y));
      const float a1 = __fadd_rn (__fmul_rn (a[k].z, a[k].z), __fmul_rn (a[k].w, a[k].w));
      float2* q0 = reinterpret_cast<float2*> (s_sqld + (u * npol) * Ms);
      q0[i] = make_float2 (a0, a1);
      // Mprime counts pol 0, as detect_skfb reads it
      if (!zero_is_valid && (a0 == 0.0f || a1 == 0.0f))
        atomicAdd (&s_zero[u], unsigned (a0 == 0.0f) + unsigned (a1 == 0.0f));
      if (two)
      {
        float2* q1 = reinterpret_cast<float2*> (s_sqld + (u * npol + 1) * Ms);
        q1[i] = make_float2 (__fadd_rn (__fmul_rn (b[k].x, b[k].x), __fmul_rn (b[k].y, b[k].y)),
                             __fadd_rn (__fmul_rn (b[k].z, b[k].z), __fmul_rn (b[k].w, b[k].w)));
      }
    }
  }
  __syncthreads ();
  if (threadIdx.x < 4 * U)
  {
    // lane = unit*4 + pol*2 + (S2 ? 1 : 0)
    const unsigned u = threadIdx.x >> 2, p = (threadIdx.x >> 1) & 1;
    const bool sq = threadIdx.x & 1;
    const bool live = u < nu && p < npol;
    const float* xf = s_sqld + (live ? u * npol + p : 0) * Ms;
    const float4* x = reinterpret_cast<const float4*> (xf);
    const unsigned nq = M / 4;
    double acc = 0.0;
    unsigned i = 0;
    if (nq >= 4)
    {
      float4 q[4];
#pragma unroll
      for (int k = 0; k < 4; k++) q[k] = x[k];
      for (i = 4; i + 4 <= nq; i += 4)
      {
        double t[16];
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
          t[4 * k] = double (sq ? __fmul_rn (q[k].x, q[k].x) : q[k].x);
          t[4 * k + 1] = double (sq ? __fmul_rn (q[k].y, q[k].y) : q[k].y);
          t[4 * k + 2] = double (sq ? __fmul_rn (q[k].z, q[k].z) : q[k].z);
          t[4 * k + 3] = double (sq ? __fmul_rn (q[k].w, q[k].w) : q[k].w);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = x[i + k];
#pragma unroll
        for (int k = 0; k < 16; k++) acc = __dadd_rn (acc, t[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
      {
        acc = __dadd_rn (acc, double (sq ? __fmul_rn (q[k].x, q[k].x) : q[k].x));
        acc = __dadd_rn (acc, double (sq ? __fmul_rn (q[k].y, q[k].y) : q[k].y));
        acc = __dadd_rn (acc, double (sq ? __fmul_rn (q[k].z, q[k].z) : q[k].z));
        acc = __dadd_rn (acc, double (sq ? __fmul_rn (q[k].w, q[k].w) : q[k].w));
      }
    }
    for (unsigned jj = 4 * i; jj < M; jj++)
      acc = __dadd_rn (acc, double (sq ? __fmul_rn (xf[jj], xf[jj]) : xf[jj]));
    if (live) s_sum[u][p][sq] = acc;
  }
  __syncthreads ();
  if (threadIdx.x < nu)
  {
    const unsigned u = threadIdx.x;
    const uint64_t unit = (part0 + u) * nchan + c;
    const unsigned Mprime = M - s_zero[u];
    bool zap = false;
    if (Mprime > 0)
    {
      zap = true;
      if (Mprime > 2)
      {
        // Equation (8) of Nita & Gary (2010b), as detect_skfb evaluates it in float
        const float M_fac = __fdiv_rn (float (Mprime * Nd + 1), float (Mprime - 1));
        zap = false;
        for (unsigned p = 0; p < npol; p++)
        {
          const float S1 = __double2float_rn (s_sum[u][p][0]);
          const float S2 = __double2float_rn (s_sum[u][p][1]);
          const float r = __fdiv_rn (S2, __fmul_rn (S1, S1));
          const float V = __fmul_rn (M_fac, __fsub_rn (__fmul_rn (float (Mprime), r), 1.0f));
          if (V > upper || V < lower) zap = true;
        }
      }
    }
    if (sums)
      for (unsigned p = 0; p < npol; p++)
      {
        sums[2 * (unit * npol + p)] = __double2float_rn (s_sum[u][p][0]);
        sums[2 * (unit * npol + p) + 1] = __double2float_rn (s_sum[u][p][1]);
      }
    if (counts) counts[unit] = Mprime;
    if (mask) mask[unit] = zap ? 1 : 0;
    if (zap && nzap) atomicAdd (nzap, 1ull);
    s_zap[u] = zap;
  }
  __syncthreads ();
  // zero the zapped blocks; each thread overwrites exactly the float4s it wrote through
  if (!out) return;
  const float4 zero = make_float4 (0.f, 0.f, 0.f, 0.f);
  for (unsigned f = threadIdx.x; f < total; f += SK_THREADS)
    if (s_zap[f / n4])
    {
      __stcs (dst0 + f, zero);
      if (two) __stcs (dst1 + f, zero);
    }
}

__global__ void k_unpack8 (const uint8_t* __restrict__ in, const uint64_t ndat,
                           const unsigned nchan, const unsigned npol, const unsigned ndim,
                           const float* __restrict__ lut, float* __restrict__ out,
                           const uint64_t span)
{
  __shared__ float s_lut[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s_lut[i] = lut[i];
  __syncthreads ();
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat) return;
  const uint8_t* src = in + (t * nchan + c) * npol * ndim;
  for (unsigned p = 0; p < npol; p++)
    for (unsigned d = 0; d < ndim; d++)
      out[(uint64_t (c) * npol + p) * span + t * ndim + d] = s_lut[src[p * ndim + d]];
}

__global__ void k_unpack16 (const int16_t* __restrict__ in, const uint64_t ndat,
                            const unsigned nchan, const unsigned npol, const unsigned ndim,
                            const int offset_binary, float* __restrict__ out,
                            const uint64_t span)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat) return;
  const int16_t* src = in + (t * nchan + c) * npol * ndim;
  for (unsigned p = 0; p < npol; p++)
    for (unsigned d = 0; d < ndim; d++)
    {
      short v = src[p * ndim + d];
      if (offset_binary) v = short (v ^ 0x8000);
      out[(uint64_t (c) * npol + p) * span + t * ndim + d] = __fadd_rn (float (v), 0.5f);
    }
}

// The unpackers for dual-polarisation complex samples: one word per sample,
// both polarisations unpacked together, an affine 8-bit table computed instead
// of looked up (a warp's lookups fall in few banks at a time).  UNPACK_T
// samples per thread keep that many loads in flight.  Bound by HBM: 17.0 us
// before, 7.9 us now for 2^21 samples (42 MB).
constexpr int UNPACK_T = 4;

template <int KIND, bool AFFINE>
__global__ void __launch_bounds__ (256)
k_unpack_pair (const typename RawPair<KIND>::T* __restrict__ in, const uint64_t ndat,
               const unsigned nchan, const float* __restrict__ lut, const float scale,
               const int offset_binary, float2* __restrict__ out, const uint64_t span)
{
  __shared__ float s_lut[KIND == IN_INT8 && !AFFINE ? 256 : 1];
  if constexpr (KIND == IN_INT8 && !AFFINE)
  {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_lut[i] = lut[i];
    __syncthreads ();
  }
  const UnpackPair u {s_lut, scale, offset_binary ? 0u : 0x80008000u};
  const uint64_t t0 = uint64_t (blockIdx.x) * (256 * UNPACK_T) + threadIdx.x;
  const unsigned c = blockIdx.y;
  typename RawPair<KIND>::T w[UNPACK_T];
#pragma unroll
  for (int k = 0; k < UNPACK_T; k++)
    if (t0 + 256 * k < ndat) w[k] = __ldg (in + (t0 + 256 * k) * nchan + c);
#pragma unroll
  for (int k = 0; k < UNPACK_T; k++)
    if (t0 + 256 * k < ndat)
    {
      const C2 x = unpack_pair<KIND, AFFINE> (w[k], u);
      float2* o = out + uint64_t (c) * 2 * span + t0 + 256 * k;
      o[0] = make_float2 (x.re.x, x.im.x);
      o[span] = make_float2 (x.re.y, x.im.y);
    }
}

__global__ void k_detect (const float2* __restrict__ in, const uint64_t in_span,
                          const uint64_t ndat, const int state, float* __restrict__ out,
                          const uint64_t out_span)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat) return;
  const float2 p = in[(uint64_t (c) * 2) * in_span + t];
  const float2 q = in[(uint64_t (c) * 2 + 1) * in_span + t];
  float v[4];
  detect_values (state, 2, p, q, v);
  const int nout = detect_nout (state);
  for (int k = 0; k < nout; k++)
    out[(uint64_t (c) * nout + k) * out_span + t] = v[k];
}

// Fold::Engine::fold on detected FPT floats (ndim 1): a warp takes
// 32 * FOLD_K consecutive samples of NP products of one channel (all of them
// when there are 1, 2 or 4; otherwise one per blockIdx.z), so that
// RowFold sums whole sets of rows.  Bound by issue and by the
// latency of its loads.
constexpr int FOLD_K = 8;

template <int NP, bool LONG>
__global__ void __launch_bounds__ (128)
k_fold (const float* __restrict__ in, const uint64_t in_span, const uint64_t ndat,
        const unsigned npol, const FoldView fv)
{
  using RF = RowFold<NP, FOLD_K>;
  __shared__ __align__ (16) float s_fold[LONG ? 4 * RF::WORDS : 4];
  const unsigned lane = threadIdx.x & 31;
  const uint64_t t0 = (uint64_t (blockIdx.x) * 4 + (threadIdx.x >> 5)) * (32 * FOLD_K) + lane;
  const unsigned c = blockIdx.y;
  for (unsigned z = blockIdx.z; z < npol / NP; z += gridDim.z)
  {
    const uint64_t row0 = uint64_t (c) * npol + z * NP;
    RF rf (s_fold + (LONG ? (threadIdx.x >> 5) * RF::WORDS : 0), fv.profiles + row0 * fv.stride, fv.stride,
           row0 == 0 ? fv.hits : nullptr);
    float v[FOLD_K][NP];
  #pragma unroll
    for (int k = 0; k < FOLD_K; k++)
  #pragma unroll
      for (int p = 0; p < NP; p++)
        v[k][p] = t0 + 32 * k < ndat ? __ldg (in + (row0 + p) * in_span + t0 + 32 * k) : 0.f;
      unsigned col[FOLD_K];
#pragma unroll
    for (int k = 0; k < FOLD_K; k++) col[k] = fold_column (fv, t0 + 32 * k < ndat, t0 + 32 * k);
#pragma unroll
    for (int k = 0; k < FOLD_K; k++)
    {
      if (!__any_sync (FULL, col[k] != NO_COLUMN)) continue;
      if constexpr (LONG)
        rf.put (col[k], v[k]);
      else
        fold_row<NP> (col[k], v[k], rf.prof, rf.stride, rf.hits);
    }
    if constexpr (LONG) rf.flush ();
  }
}

// SampleDelay::transformation (SampleDelay.C:247-298) fused with detection and
// the fold: output sample t of channel c is voltage t + applied[c] of that
// channel (rows [chan][pol] of span values).
template <int NOUT>
__global__ void k_delay_fold (const float2* __restrict__ v, const uint64_t span,
                              const int* __restrict__ applied, const uint64_t ndat,
                              const unsigned npol, const FoldView fv)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  const bool ok = t < ndat;
  float2 p = make_float2 (0.f, 0.f), q = make_float2 (0.f, 0.f);
  if (ok)
  {
    const uint64_t i = t + uint64_t (__ldg (applied + c));
    p = v[(uint64_t (c) * npol) * span + i];
    if (npol == 2) q = v[(uint64_t (c) * npol + 1) * span + i];
  }
  if (!__any_sync (FULL, ok)) return;
  const unsigned col = fold_column (fv, ok, t);
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  detect_values (fv.state, npol, p, q, d);
  fold_row<NOUT> (col, d, fv.profiles + uint64_t (c) * NOUT * fv.stride, fv.stride,
                  c == 0 ? fv.hits : nullptr);
}

// SpectralKurtosis::detect_skfb (SpectralKurtosis.C:1105-1222) from sums
// already formed: per (part, chan), Mprime = counts (M when counts is null);
// none counted leaves the mask as it is, one or two zap, otherwise the
// estimator of each polarisation is tested in float as the reference does.
// Zapped cells are set to 1 (others are left alone, as the reference leaves
// them to reset_mask).
__global__ void k_sk_detect (const float* __restrict__ sums, const unsigned* __restrict__ counts,
                             const uint64_t ncell, const unsigned npol, const unsigned M,
                             const unsigned Nd, const float lower, const float upper,
                             uint8_t* __restrict__ mask, unsigned long long* __restrict__ nzap)
{
  const uint64_t unit = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  if (unit >= ncell) return;
  const unsigned Mprime = counts ? counts[unit] : M;
  if (Mprime == 0) return;
  bool zap = true;
  if (Mprime > 2)
  {
    const float M_fac = __fdiv_rn (float (Mprime * Nd + 1), float (Mprime - 1));
    zap = false;
    for (unsigned p = 0; p < npol; p++)
    {
      const float S1 = sums[2 * (unit * npol + p)];
      const float S2 = sums[2 * (unit * npol + p) + 1];
      const float r = __fdiv_rn (S2, __fmul_rn (S1, S1));
      const float V = __fmul_rn (M_fac, __fsub_rn (__fmul_rn (float (Mprime), r), 1.0f));
      if (V > upper || V < lower) zap = true;
    }
  }
  if (zap)
  {
    mask[unit] = 1;
    if (nzap) atomicAdd (nzap, 1ull);
  }
}

// SpectralKurtosis::compute (SpectralKurtosis.C:674-798) for blocks of M
// samples every `stride` samples (Resolution::prepare with noverlap =
// M / stride, :251-281): one thread per (block, chan, pol, S1 or S2) adds the
// block's values in order in double, as the reference does; S2 adds the
// float square of each sqld.  counts (pol 0's S1 thread) as the reference's
// sum weights.  Blocks overlap, so each sample is read noverlap times; the
// non-overlapping case has its own faster kernel (k_sk).
__global__ void k_sk_sums_strided (const float2* __restrict__ in, const uint64_t span,
                                   const uint64_t nblk, const uint64_t stride,
                                   const unsigned nchan, const unsigned npol, const unsigned M,
                                   const int zero_is_valid, float* __restrict__ sums,
                                   unsigned* __restrict__ counts)
{
  const uint64_t idx = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t total = nblk * nchan * npol * 2;
  if (idx >= total) return;
  const unsigned sq = unsigned (idx & 1);
  const unsigned p = unsigned ((idx >> 1) % npol);
  const uint64_t bc = (idx >> 1) / npol;
  const unsigned c = unsigned (bc % nchan);
  const uint64_t b = bc / nchan;
  const float2* x = in + (uint64_t (c) * npol + p) * span + b * stride;
  double acc = 0.0;
  unsigned n = 0;
  for (unsigned i = 0; i < M; i++)
  {
    const float2 v = x[i];
    const float d = __fadd_rn (__fmul_rn (v.x, v.x), __fmul_rn (v.y, v.y));
    if (zero_is_valid || d != 0.0f)
    {
      acc = __dadd_rn (acc, double (sq ? __fmul_rn (d, d) : d));
      n++;
    }
  }
  const uint64_t unit = b * nchan + c;
  sums[2 * (unit * npol + p) + sq] = __double2float_rn (acc);
  if (counts && p == 0 && sq == 0) counts[unit] = n;
}

// SpectralKurtosis::tscrunch_sums (SpectralKurtosis.C:917-986): coarse part q
// takes the fine parts q*offset + isum*offset, isum < nsum, adding the float
// sums and the counts in that order (the reference's indexing, kept as it is)
__global__ void k_sk_tscrunch (const float* __restrict__ sums, const unsigned* __restrict__ counts,
                               const uint64_t npart, const unsigned nchan, const unsigned npol,
                               const unsigned nsum, const unsigned offset,
                               float* __restrict__ osums, unsigned* __restrict__ ocounts)
{
  const uint64_t idx = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t per = uint64_t (nchan) * npol * 2;
  if (idx >= npart * per) return;
  const uint64_t q = idx / per, e = idx % per;
  float acc = sums[(q * offset) * per + e];
  for (unsigned isum = 1; isum < nsum; isum++)
    acc = __fadd_rn (acc, sums[(q * offset + uint64_t (isum) * offset) * per + e]);
  osums[idx] = acc;
  // the counts: one per (part, chan), from the threads of pol 0's S1
  if (e % (npol * 2) == 0)
  {
    const unsigned c = unsigned (e / (npol * 2));
    unsigned n = counts ? counts[(q * offset) * nchan + c] : 0;
    for (unsigned isum = 1; isum < nsum && counts; isum++)
      n += counts[(q * offset + uint64_t (isum) * offset) * nchan + c];
    if (ocounts) ocounts[q * nchan + c] = n;
  }
}

// SpectralKurtosis::detect_skfb (SpectralKurtosis.C:1105-1222) at one
// resolution: thresholds from a table of (count, lower, upper) sorted by
// count (get_limits of each count present); a zapped coarse cell flags nflag
// fine cells, flag_step fine parts apart, starting at q * flag_offset.
__global__ void k_sk_detect_skfb (const float* __restrict__ sums, const unsigned* __restrict__ counts,
                                  const uint64_t npart, const unsigned nchan, const unsigned npol,
                                  const unsigned Nd, const unsigned* __restrict__ lim_count,
                                  const float2* __restrict__ lim, const unsigned nlim,
                                  const unsigned nflag, const unsigned flag_step,
                                  const unsigned flag_offset, uint8_t* __restrict__ mask,
                                  unsigned long long* __restrict__ nzap)
{
  const uint64_t unit = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  if (unit >= npart * nchan) return;
  const unsigned Mprime = counts[unit];
  if (Mprime == 0) return;
  bool zap = true;
  if (Mprime > 2)
  {
    unsigned lo = 0, hi = nlim;
    while (lo + 1 < hi)
    {
      const unsigned mid = (lo + hi) / 2;
      if (lim_count[mid] <= Mprime) lo = mid; else hi = mid;
    }
    const float2 L = lim[lo];       // (lower, upper); the table holds every count present
    const float M_fac = __fdiv_rn (float (Mprime * Nd + 1), float (Mprime - 1));
    zap = false;
    for (unsigned p = 0; p < npol; p++)
    {
      const float S1 = sums[2 * (unit * npol + p)];
      const float S2 = sums[2 * (unit * npol + p) + 1];
      const float r = __fdiv_rn (S2, __fmul_rn (S1, S1));
      const float V = __fmul_rn (M_fac, __fsub_rn (__fmul_rn (float (Mprime), r), 1.0f));
      if (V > L.y || V < L.x) zap = true;
    }
  }
  if (!zap) return;
  if (nzap) atomicAdd (nzap, 1ull);
  const uint64_t q = unit / nchan;
  const unsigned c = unsigned (unit % nchan);
  for (unsigned f = 0; f < nflag; f++)
    mask[(q * flag_offset + uint64_t (f) * flag_step) * nchan + c] = 1;
}

// SpectralKurtosis::mask with overlapping blocks (SpectralKurtosis.C:1465-
// 1566): the reference copies (or zeroes) part after part, M samples each,
// parts `offset` apart, so a sample keeps the decision of the last part that
// covers it: part min(t / offset, npart - 1), mask row part + nskip; the
// input is read from idat_start on.
__global__ void k_sk_mask_overlap (const uint8_t* __restrict__ mask, const float2* __restrict__ in,
                                   const uint64_t in_span, float2* __restrict__ out,
                                   const uint64_t out_span, const uint64_t ndat_out,
                                   const unsigned nchan, const unsigned npol,
                                   const unsigned offset, const uint64_t npart,
                                   const uint64_t nskip, const uint64_t idat_start)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat_out) return;
  const uint64_t part = min (t / offset, npart - 1);
  const bool zap = __ldg (mask + (part + nskip) * nchan + c) != 0;
  for (unsigned p = 0; p < npol; p++)
  {
    const uint64_t r = uint64_t (c) * npol + p;
    out[r * out_span + t] = zap ? make_float2 (0.f, 0.f) : in[r * in_span + idat_start + t];
  }
}

// SpectralKurtosis::mask (SpectralKurtosis.C:1465-1566): out = in, with the
// blocks whose mask is set zeroed (in place when out == in: only those are
// written).
__global__ void k_sk_mask (const uint8_t* __restrict__ mask, const float2* in, const uint64_t in_span,
                           float2* out, const uint64_t out_span, const uint64_t ndat,
                           const unsigned nchan, const unsigned npol, const unsigned M)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat) return;
  const bool zap = __ldg (mask + (t / M) * nchan + c) != 0;
  const bool inplace = in == out && in_span == out_span;
  for (unsigned p = 0; p < npol; p++)
  {
    const uint64_t r = uint64_t (c) * npol + p;
    if (zap) out[r * out_span + t] = make_float2 (0.f, 0.f);
    else if (!inplace) out[r * out_span + t] = in[r * in_span + t];
  }
}

// Convolution's zero-DM output (Convolution.C:175-193, 789-796) for the
// pipeline: input sample first + t of every (chan, pol), unpacked, into
// out[(c*npol + p)*span + t]
template <int KIND>
__global__ void k_zero_dm (const InputView in, const float* __restrict__ lut, const uint64_t first,
                           const uint64_t n, float2* __restrict__ out, const uint64_t span)
{
  __shared__ float s_lut[256];
  if constexpr (KIND == IN_INT8) load_lut (in, lut, s_lut);
  __syncthreads ();
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const unsigned row = blockIdx.y, c = row / in.npol, p = row % in.npol;
  out[uint64_t (row) * span + t] = fetch<KIND> (in, s_lut, c, p, first + t);
}

// SpectralKurtosis::mask (SpectralKurtosis.C:1465-1566) applied to other
// voltages than the statistics came from (the dedispersed ones, when the
// statistics are of the zero-DM input): block t / M of channel c is zeroed
// in every polarisation where mask[(t / M) * nchan + c] is set.
__global__ void k_sk_apply (const uint8_t* __restrict__ mask, float2* __restrict__ v,
                            const uint64_t span, const uint64_t ndat, const unsigned nchan,
                            const unsigned npol, const unsigned M)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  if (t >= ndat || !__ldg (mask + (t / M) * nchan + c)) return;
  for (unsigned p = 0; p < npol; p++) v[(uint64_t (c) * npol + p) * span + t] = make_float2 (0.f, 0.f);
}

// Detection and Fold::fold of data with zeroed samples (Fold.C:895-930,
// zeroed_samples): every sample is added to its bin, and a hit is counted
// for each channel whose first detected value of the first polarisation is
// non-zero -- into the one hits array shared by all channels.
template <int NOUT>
__global__ void k_zeroed_fold (const float2* __restrict__ v, const uint64_t span,
                               const uint64_t ndat, const unsigned npol, const FoldView fv)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned c = blockIdx.y;
  const bool ok = t < ndat;
  if (!__any_sync (FULL, ok)) return;
  float2 p = make_float2 (0.f, 0.f), q = make_float2 (0.f, 0.f);
  if (ok)
  {
    p = v[(uint64_t (c) * npol) * span + t];
    if (npol == 2) q = v[(uint64_t (c) * npol + 1) * span + t];
  }
  unsigned col = fold_column (fv, ok, t);
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  detect_values (fv.state, npol, p, q, d);
  // a zeroed sample adds nothing to the profile and counts no hit
  if (d[0] == 0.f) col = NO_COLUMN;
  fold_row<NOUT> (col, d, fv.profiles + uint64_t (c) * NOUT * fv.stride, fv.stride, fv.hits);
}

// Segment holding sample t, found by a whole warp: each round probes 32
// evenly spaced starts at once (two dependent loads for up to 1024 segments,
// where a binary search takes ten).
__device__ __forceinline__ int warp_seg_search (const FoldSegment* __restrict__ segs, int nseg,
                                                uint64_t t)
{
  const int lane = threadIdx.x & 31;
  int lo = 0, len = nseg;
  while (len > 1)
  {
    const int step = (len + 31) / 32;
    const int off = lane * step;
    const bool le = off < len && (off == 0 || __ldg (&segs[lo + off].start) <= t);
    const int j = 31 - __clz (__ballot_sync (FULL, le));
    lo += j * step;
    len = min (step, len - j * step);
  }
  return lo;
}

// The column warp_fold_bin would give each sample.  A warp takes
// COLPLAN_SAMPLES consecutive samples, each lane four at a time (one 16-byte
// store): one search for the first sample, further ones in groups that cross
// a segment boundary, and a lane's samples advance m by dm within a segment.
// Bound by latency (the search, the segment loads and the double chain), so
// the serial chain per warp is kept short: one sample per lane and 32 groups
// per warp took 37.6 us for 10 M samples and 7.7 us for 60 k; this takes 24.2 and 3.9 us.
// (Adding powers of two instead of the 64-bit conversions: 31.0 us.)
// Stepping lane by lane through runs of one-sample segments took 33 us for
// 860 segments in 6 M samples, the search per lane 16 us.
constexpr int COLPLAN_SAMPLES = 512;

__global__ void __launch_bounds__ (256)
k_colplan (const FoldSegment* __restrict__ segs, const int nseg, const uint64_t ndat,
           const unsigned nbin, unsigned* __restrict__ cols)
{
  const int lane = threadIdx.x & 31;
  const uint64_t w0 = (uint64_t (blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32)
                      * COLPLAN_SAMPLES;
  if (w0 >= ndat) return;             // whole warps
  int s = warp_seg_search (segs, nseg, w0);
  const double fbin = double (nbin);
#pragma unroll 1
  for (int g = 0; g < COLPLAN_SAMPLES; g += 128)
  {
    const uint64_t t0 = w0 + unsigned (g) + 4 * lane;
    // where the group crosses segments (hundreds of one-sample ones can follow
    // one another) each lane searches for its own
    const uint64_t last = w0 + unsigned (g) + 127;
    if (s + 1 < nseg && __ldg (&segs[s + 1].start) <= last)
    {
      const int e = s + warp_seg_search (segs + s, nseg - s, last);
      s += seg_search (segs + s, e - s + 1, t0);
    }
    unsigned c[4];
    int64_t m = 0, dm = 0;
    double gr = 0;
    unsigned base = 0;
    uint64_t next = 0;                // the segment's end; 0: none loaded yet
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
      const uint64_t t = t0 + i;
      if (t >= next)
      {
        if (next) s++;
        while (s + 1 < nseg && __ldg (&segs[s + 1].start) <= t) s++;
        next = s + 1 < nseg ? __ldg (&segs[s + 1].start) : ~uint64_t (0);
        dm = __ldg (&segs[s].dm);
        m = __ldg (&segs[s].m0) + int64_t (t - __ldg (&segs[s].start)) * dm;
        gr = __ldg (&segs[s].g);
        base = __ldg (&segs[s].base);
      }
      const unsigned bin = __double2uint_rz (__dmul_rn (__dmul_rn (double (m), gr), fbin));
      c[i] = (base == FOLD_SKIP || bin >= nbin) ? NO_COLUMN : base + bin;
      m += dm;
    }
    if (t0 + 4 <= ndat)
      *reinterpret_cast<uint4*> (cols + t0) = make_uint4 (c[0], c[1], c[2], c[3]);
    else
      for (int i = 0; i < 4; i++)
        if (t0 + i < ndat) cols[t0 + i] = c[i];
    s = __shfl_sync (FULL, s, 31);
  }
}

__global__ void k_binplan (const FoldSegment* __restrict__ segs, const int nseg,
                           const uint64_t ndat, const unsigned nbin, uint32_t* __restrict__ out)
{
  const uint64_t t = uint64_t (blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= ndat) return;
  out[t] = fold_bin (segs, nseg, t, nbin);
}

} // namespace

uint64_t kernel_launches () { return g_launches.load (); }

unsigned pass_tables_count (unsigned n)
{
  switch (n)
  {
    case 64: return pass_tables_size (64);
    case 128: return pass_tables_size (128);
    case 256: return pass_tables_size (256);
    case 512: return pass_tables_size (512);
    case 1024: return pass_tables_size (1024);
    case 2048: return pass_tables_size (2048);
    case 4096: return pass_tables_size (4096);
    case 8192: return pass_tables_size (8192);
    default: return 0;
  }
}

// w_{Ns R}^{a r} rounded once from double precision, [r-1][a] per pass
void make_pass_tables (unsigned n, float2* out, unsigned capacity)
{
  const int N = int (n);
  for (int p = 1; p < stockham_npass (N); p++)
  {
    const int Ns = stockham_ns (N, p), R = stockham_radix (N, p);
    const int off = pass_table_offset (N, p);
    for (int r = 1; r < R; r++)
      for (int a = 0; a < Ns; a++)
      {
        const unsigned idx = unsigned (off + (r - 1) * Ns + a);
        if (idx >= capacity) return;
        const double ang = -2.0 * 3.14159265358979323846 * double (a) * r / (double (Ns) * R);
        out[idx] = make_float2 (float (cos (ang)), float (sin (ang)));
      }
  }
}

cudaError_t launch_build_chirp (float2* H, const double* d_chan_freq, const double* d_coeff,
                                const double* d_frac_us, unsigned nchan, unsigned nfft,
                                unsigned n1, unsigned n2, double binwidth, double half_chanwidth,
                                int swap_halves, int chirp_mode, float scale, cudaStream_t st)
{
  const dim3 grid ((nfft + 255) / 256, nchan);
  g_launches++;
  k_build_chirp<<<grid, 256, 0, st>>> (H, d_chan_freq, d_coeff, d_frac_us, nfft, n1, n2,
                                        binwidth, half_chanwidth, swap_halves, chirp_mode, scale);
  return cudaGetLastError ();
}

cudaError_t launch_permute_response (float2* H, const float2* src, unsigned nchan, unsigned n1,
                                     unsigned n2, cudaStream_t st)
{
  const uint64_t N = uint64_t (n1) * n2;
  g_launches++;
  k_permute<<<dim3 (unsigned ((N + 255) / 256), nchan), 256, 0, st>>> (H, src, n1, n2, 0);
  return cudaGetLastError ();
}

cudaError_t launch_unpermute_response (float2* dst, const float2* H, unsigned nchan, unsigned n1,
                                       unsigned n2, cudaStream_t st)
{
  const uint64_t N = uint64_t (n1) * n2;
  g_launches++;
  k_permute<<<dim3 (unsigned ((N + 255) / 256), nchan), 256, 0, st>>> (dst, H, n1, n2, 1);
  return cudaGetLastError ();
}

namespace {
template <int NSUB>
cudaError_t run_filterbank (const InputView& in, const float* d_lut, uint64_t nblk, float scale,
                            float2* out, uint64_t out_span, cudaStream_t st,
                            const KernelClock* clk)
{
  const dim3 grid (unsigned ((nblk + 127) / 128), in.npol, in.nchan);
  ClockScope cs (clk, KK_FILTERBANK, st);
  if (in.kind == IN_INT8)
    k_filterbank<NSUB, IN_INT8><<<grid, 128, 0, st>>> (in, d_lut, nblk, scale, out, out_span);
  else if (in.kind == IN_INT16)
    k_filterbank<NSUB, IN_INT16><<<grid, 128, 0, st>>> (in, d_lut, nblk, scale, out, out_span);
  else
    k_filterbank<NSUB, IN_FLOAT><<<grid, 128, 0, st>>> (in, d_lut, nblk, scale, out, out_span);
  return cudaGetLastError ();
}
// multiprocessors of the current device, asked for once per device
cudaError_t sm_count (int* n)
{
  static std::atomic<int> known[32] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess) return e;
  if (dev < 32 && known[dev].load ())
  {
    *n = known[dev].load ();
    return cudaSuccess;
  }
  e = cudaDeviceGetAttribute (n, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess && dev < 32) known[dev].store (*n);
  return e;
}

template <int NSUB, int KIND, bool TWO>
cudaError_t run_filterbank_warp_t (const InputView& in, const float* d_lut, uint64_t nblk,
                                   float scale, float2* out, uint64_t out_span, cudaStream_t st)
{
  using F = FbWarp<NSUB>;
  auto kern = k_filterbank_warp<NSUB, KIND, TWO>;
  int nsm = 0;
  cudaError_t e = sm_count (&nsm);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int (F::SMEM));
  if (e != cudaSuccess) return e;
  const unsigned pols = TWO ? 2 : 1, nbt = F::NB / pols;
  const uint64_t per_row = (nblk + nbt - 1) / nbt;
  const uint64_t ntile = per_row * in.nchan * in.npol / pols;
  const unsigned grid = unsigned (std::min<uint64_t> (ntile, 2 * uint64_t (nsm)));
  kern<<<grid, FBW_WARPS * 32, F::SMEM, st>>> (in, d_lut, nblk, scale, out, out_span, per_row, ntile);
  return cudaGetLastError ();
}

template <int NSUB>
cudaError_t run_filterbank_warp (const InputView& in, const float* d_lut, uint64_t nblk, float scale,
                                 float2* out, uint64_t out_span, cudaStream_t st,
                                 const KernelClock* clk)
{
  ClockScope cs (clk, KK_FILTERBANK, st);
  if constexpr (NSUB <= 512)
    if (in.npol == 2 && in.kind != IN_FLOAT)
      return in.kind == IN_INT8
             ? run_filterbank_warp_t<NSUB, IN_INT8, true> (in, d_lut, nblk, scale, out, out_span, st)
             : run_filterbank_warp_t<NSUB, IN_INT16, true> (in, d_lut, nblk, scale, out, out_span, st);
  if (in.kind == IN_INT8)
    return run_filterbank_warp_t<NSUB, IN_INT8, false> (in, d_lut, nblk, scale, out, out_span, st);
  if (in.kind == IN_INT16)
    return run_filterbank_warp_t<NSUB, IN_INT16, false> (in, d_lut, nblk, scale, out, out_span, st);
  return run_filterbank_warp_t<NSUB, IN_FLOAT, false> (in, d_lut, nblk, scale, out, out_span, st);
}

template <int NSUB>
cudaError_t run_filterbank_smem (const InputView& in, const float* d_lut, const float2* ptab,
                                 uint64_t nblk, float scale, float2* out, uint64_t out_span,
                                 cudaStream_t st, const KernelClock* clk)
{
  constexpr int F = FB_THREADS / stockham_threads (NSUB);
  const unsigned bpc = F / in.npol;
  const size_t smem = (size_t (F) * (spad_size (NSUB) + 1) + pass_tables_size (NSUB)) *
                      sizeof (float2);
  const dim3 grid (unsigned ((nblk + bpc - 1) / bpc), in.nchan);
  ClockScope cs (clk, KK_FILTERBANK, st);
  cudaError_t e;
  if (in.kind == IN_INT8)
  {
    e = cudaFuncSetAttribute (k_filterbank_smem<NSUB, IN_INT8>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
    if (e == cudaSuccess)
      k_filterbank_smem<NSUB, IN_INT8><<<grid, FB_THREADS, smem, st>>> (in, d_lut, ptab, nblk,
                                                                        scale, out, out_span);
  }
  else if (in.kind == IN_INT16)
  {
    e = cudaFuncSetAttribute (k_filterbank_smem<NSUB, IN_INT16>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
    if (e == cudaSuccess)
      k_filterbank_smem<NSUB, IN_INT16><<<grid, FB_THREADS, smem, st>>> (in, d_lut, ptab, nblk,
                                                                         scale, out, out_span);
  }
  else
  {
    e = cudaFuncSetAttribute (k_filterbank_smem<NSUB, IN_FLOAT>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, int (smem));
    if (e == cudaSuccess)
      k_filterbank_smem<NSUB, IN_FLOAT><<<grid, FB_THREADS, smem, st>>> (in, d_lut, ptab, nblk,
                                                                         scale, out, out_span);
  }
  if (e != cudaSuccess) return e;
  return cudaGetLastError ();
}
} // namespace

cudaError_t launch_filterbank (const InputView& in, const float* d_lut, unsigned nsub,
                               uint64_t nblk, float scale, float2* out, uint64_t out_span,
                               cudaStream_t st, const KernelClock* clk, const float2* ptab)
{
  if (nblk == 0) return cudaSuccess;
  // up to 64 channels the one-thread-per-block register transform is faster;
  // 128 to 1024 fit a warp with 32 points per thread, more need the block
  if (filterbank_uses_tables (nsub) && !ptab) return cudaErrorInvalidValue;
  if (nsub >= 128)
  {
    switch (nsub)
    {
      case 128: return run_filterbank_warp<128> (in, d_lut, nblk, scale, out, out_span, st, clk);
      case 256: return run_filterbank_warp<256> (in, d_lut, nblk, scale, out, out_span, st, clk);
      case 512: return run_filterbank_warp<512> (in, d_lut, nblk, scale, out, out_span, st, clk);
      case 1024: return run_filterbank_warp<1024> (in, d_lut, nblk, scale, out, out_span, st, clk);
      case 2048: return run_filterbank_smem<2048> (in, d_lut, ptab, nblk, scale, out, out_span, st, clk);
      case 4096: return run_filterbank_smem<4096> (in, d_lut, ptab, nblk, scale, out, out_span, st, clk);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (nsub)
  {
    case 4: return run_filterbank<4> (in, d_lut, nblk, scale, out, out_span, st, clk);
    case 8: return run_filterbank<8> (in, d_lut, nblk, scale, out, out_span, st, clk);
    case 16: return run_filterbank<16> (in, d_lut, nblk, scale, out, out_span, st, clk);
    case 32: return run_filterbank<32> (in, d_lut, nblk, scale, out, out_span, st, clk);
    case 64: return run_filterbank<64> (in, d_lut, nblk, scale, out, out_span, st, clk);
    default: return cudaErrorInvalidValue;
  }
}

size_t sk_smem_bytes (unsigned npol, unsigned M, unsigned units)
{
  return size_t (units) * npol * sk_column (M) * sizeof (float);
}

cudaError_t launch_sk (const float2* in, uint64_t in_span, float2* out, uint64_t out_span,
                       uint64_t npart, unsigned nchan, unsigned npol, unsigned M,
                       int zero_is_valid, unsigned Nd, float lower, float upper, float* sums,
                       unsigned* counts, uint8_t* mask, unsigned long long* nzap, cudaStream_t st)
{
  if (npart == 0) return cudaSuccess;
  // as many blocks per CTA as SK_TILE holds: the sums of one occupy 4 lanes of
  // a warp, and a tile is streamed in two rounds of loads
  unsigned units = 8;
  while (units > 1 && sk_smem_bytes (npol, M, units) > SK_TILE) units /= 2;
  const size_t smem = sk_smem_bytes (npol, M, units);
  if (smem > SK_SMEM_MAX) return cudaErrorInvalidValue;
  const uint64_t nblk = (npart + units - 1) / units;
  if (nblk > 0x7fffffffull || nchan > 65535) return cudaErrorInvalidValue;
  auto kern = units == 8 ? k_sk<8> : units == 4 ? k_sk<4> : units == 2 ? k_sk<2> : k_sk<1>;
  cudaError_t e = cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int (smem));
  if (e != cudaSuccess) return e;
  g_launches++;
  kern<<<dim3 (unsigned (nblk), nchan), SK_THREADS, smem, st>>> (
      in, in_span, out, out_span, npart, nchan, npol, M, zero_is_valid, Nd, lower, upper, sums,
      counts, mask, nzap);
  return cudaGetLastError ();
}

namespace {

// dual-polarisation complex samples whose words and output values are aligned
bool unpack_as_pairs (const void* in, unsigned word, unsigned npol, unsigned ndim, const float* out,
                      uint64_t span)
{
  return npol == 2 && ndim == 2 && reinterpret_cast<uintptr_t> (in) % word == 0
         && reinterpret_cast<uintptr_t> (out) % 8 == 0 && span % 2 == 0;
}

} // namespace

cudaError_t launch_unpack8 (const uint8_t* in, uint64_t ndat, unsigned nchan, unsigned npol,
                            unsigned ndim, const float* d_lut, float lut_scale, float* out,
                            uint64_t span, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  if (unpack_as_pairs (in, 4, npol, ndim, out, span))
  {
    const dim3 grid (unsigned ((ndat + 256 * UNPACK_T - 1) / (256 * UNPACK_T)), nchan);
    auto k = lut_scale != 0.f ? k_unpack_pair<IN_INT8, true> : k_unpack_pair<IN_INT8, false>;
    k<<<grid, 256, 0, st>>> (reinterpret_cast<const unsigned*> (in), ndat, nchan, d_lut, lut_scale, 0,
                             reinterpret_cast<float2*> (out), span / 2);
    return cudaGetLastError ();
  }
  k_unpack8<<<dim3 (unsigned ((ndat + 255) / 256), nchan), 256, 0, st>>> (
      in, ndat, nchan, npol, ndim, d_lut, out, span);
  return cudaGetLastError ();
}

cudaError_t launch_unpack16 (const int16_t* in, uint64_t ndat, unsigned nchan, unsigned npol,
                             unsigned ndim, int offset_binary, float* out, uint64_t span,
                             cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  if (unpack_as_pairs (in, 8, npol, ndim, out, span))
  {
    const dim3 grid (unsigned ((ndat + 256 * UNPACK_T - 1) / (256 * UNPACK_T)), nchan);
    k_unpack_pair<IN_INT16, false><<<grid, 256, 0, st>>> (
        reinterpret_cast<const uint2*> (in), ndat, nchan, nullptr, 0.f, offset_binary,
        reinterpret_cast<float2*> (out), span / 2);
    return cudaGetLastError ();
  }
  k_unpack16<<<dim3 (unsigned ((ndat + 255) / 256), nchan), 256, 0, st>>> (
      in, ndat, nchan, npol, ndim, offset_binary, out, span);
  return cudaGetLastError ();
}

cudaError_t launch_detect (const float2* in, uint64_t in_span, uint64_t ndat, unsigned nchan,
                           int state, float* out, uint64_t out_span, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  k_detect<<<dim3 (unsigned ((ndat + 255) / 256), nchan), 256, 0, st>>> (in, in_span, ndat,
                                                                          state, out, out_span);
  return cudaGetLastError ();
}

cudaError_t launch_fold (const float* in, uint64_t in_span, uint64_t ndat, unsigned nchan,
                         unsigned npol, const FoldView& fv, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  const unsigned gx = unsigned ((ndat + 128 * FOLD_K - 1) / (128 * FOLD_K));
  const auto run = [&] (auto kern, unsigned gz) {
    kern<<<dim3 (gx, nchan, gz), 128, 0, st>>> (in, in_span, ndat, npol, fv);
  };
  if (npol == 4)
    run (fv.long_bins ? k_fold<4, true> : k_fold<4, false>, 1);
  else if (npol == 2)
    run (fv.long_bins ? k_fold<2, true> : k_fold<2, false>, 1);
  else
    run (fv.long_bins ? k_fold<1, true> : k_fold<1, false>, std::min (npol, 65535u));
  return cudaGetLastError ();
}

cudaError_t launch_colplan (const FoldSegment* segs, int nseg, uint64_t ndat, unsigned nbin,
                            unsigned* cols, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  const uint64_t per_block = uint64_t (256 / 32) * COLPLAN_SAMPLES;
  k_colplan<<<unsigned ((ndat + per_block - 1) / per_block), 256, 0, st>>> (segs, nseg, ndat,
                                                                           nbin, cols);
  return cudaGetLastError ();
}

cudaError_t launch_delay_fold (const float2* v, uint64_t span, const int* applied, uint64_t ndat,
                               unsigned nchan, unsigned npol, const FoldView& fv, cudaStream_t st,
                               const KernelClock* clk)
{
  if (ndat == 0) return cudaSuccess;
  const dim3 grid (unsigned ((ndat + 255) / 256), nchan);
  ClockScope cs (clk, KK_INV_COLS, st);
  if (fv.nout == 1)
    k_delay_fold<1><<<grid, 256, 0, st>>> (v, span, applied, ndat, npol, fv);
  else if (fv.nout == 2)
    k_delay_fold<2><<<grid, 256, 0, st>>> (v, span, applied, ndat, npol, fv);
  else
    k_delay_fold<4><<<grid, 256, 0, st>>> (v, span, applied, ndat, npol, fv);
  return cudaGetLastError ();
}

cudaError_t launch_sk_sums_strided (const float2* in, uint64_t span, uint64_t nblk,
                                   uint64_t stride, unsigned nchan, unsigned npol, unsigned M,
                                   int zero_is_valid, float* sums, unsigned* counts,
                                   cudaStream_t st)
{
  const uint64_t total = nblk * nchan * npol * 2;
  if (total == 0) return cudaSuccess;
  g_launches++;
  k_sk_sums_strided<<<unsigned ((total + 127) / 128), 128, 0, st>>> (
      in, span, nblk, stride, nchan, npol, M, zero_is_valid, sums, counts);
  return cudaGetLastError ();
}

cudaError_t launch_sk_tscrunch (const float* sums, const unsigned* counts, uint64_t npart,
                                unsigned nchan, unsigned npol, unsigned nsum, unsigned offset,
                                float* osums, unsigned* ocounts, cudaStream_t st)
{
  const uint64_t total = npart * nchan * npol * 2;
  if (total == 0) return cudaSuccess;
  g_launches++;
  k_sk_tscrunch<<<unsigned ((total + 255) / 256), 256, 0, st>>> (sums, counts, npart, nchan, npol,
                                                                 nsum, offset, osums, ocounts);
  return cudaGetLastError ();
}

cudaError_t launch_sk_detect_skfb (const float* sums, const unsigned* counts, uint64_t npart,
                                   unsigned nchan, unsigned npol, unsigned Nd,
                                   const unsigned* lim_count, const float2* lim, unsigned nlim,
                                   unsigned nflag, unsigned flag_step, unsigned flag_offset,
                                   uint8_t* mask, unsigned long long* nzap, cudaStream_t st)
{
  const uint64_t total = npart * nchan;
  if (total == 0) return cudaSuccess;
  g_launches++;
  k_sk_detect_skfb<<<unsigned ((total + 255) / 256), 256, 0, st>>> (
      sums, counts, npart, nchan, npol, Nd, lim_count, lim, nlim, nflag, flag_step, flag_offset,
      mask, nzap);
  return cudaGetLastError ();
}

cudaError_t launch_sk_mask_overlap (const uint8_t* mask, const float2* in, uint64_t in_span,
                                    float2* out, uint64_t out_span, uint64_t ndat_out,
                                    unsigned nchan, unsigned npol, unsigned offset,
                                    uint64_t npart, uint64_t nskip, uint64_t idat_start,
                                    cudaStream_t st)
{
  if (ndat_out == 0 || npart == 0) return cudaSuccess;
  g_launches++;
  k_sk_mask_overlap<<<dim3 (unsigned ((ndat_out + 255) / 256), nchan), 256, 0, st>>> (
      mask, in, in_span, out, out_span, ndat_out, nchan, npol, offset, npart, nskip, idat_start);
  return cudaGetLastError ();
}

cudaError_t launch_sk_detect (const float* sums, const unsigned* counts, uint64_t npart,
                              unsigned nchan, unsigned npol, unsigned M, unsigned Nd, float lower,
                              float upper, uint8_t* mask, unsigned long long* nzap, cudaStream_t st)
{
  const uint64_t ncell = npart * nchan;
  if (ncell == 0) return cudaSuccess;
  g_launches++;
  k_sk_detect<<<unsigned ((ncell + 255) / 256), 256, 0, st>>> (sums, counts, ncell, npol, M, Nd,
                                                              lower, upper, mask, nzap);
  return cudaGetLastError ();
}

cudaError_t launch_sk_mask (const uint8_t* mask, const float2* in, uint64_t in_span, float2* out,
                            uint64_t out_span, uint64_t ndat, unsigned nchan, unsigned npol,
                            unsigned M, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  k_sk_mask<<<dim3 (unsigned ((ndat + 255) / 256), nchan), 256, 0, st>>> (
      mask, in, in_span, out, out_span, ndat, nchan, npol, M);
  return cudaGetLastError ();
}

cudaError_t launch_zero_dm (const InputView& in, const float* lut, uint64_t first, uint64_t n,
                            float2* out, uint64_t span, cudaStream_t st)
{
  if (n == 0) return cudaSuccess;
  g_launches++;
  const dim3 grid (unsigned ((n + 255) / 256), in.nchan * in.npol);
  if (in.kind == IN_INT8)
    k_zero_dm<IN_INT8><<<grid, 256, 0, st>>> (in, lut, first, n, out, span);
  else if (in.kind == IN_INT16)
    k_zero_dm<IN_INT16><<<grid, 256, 0, st>>> (in, lut, first, n, out, span);
  else
    k_zero_dm<IN_FLOAT><<<grid, 256, 0, st>>> (in, lut, first, n, out, span);
  return cudaGetLastError ();
}

cudaError_t launch_sk_apply (const uint8_t* mask, float2* v, uint64_t span, uint64_t ndat,
                             unsigned nchan, unsigned npol, unsigned M, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  k_sk_apply<<<dim3 (unsigned ((ndat + 255) / 256), nchan), 256, 0, st>>> (mask, v, span, ndat,
                                                                            nchan, npol, M);
  return cudaGetLastError ();
}

cudaError_t launch_zeroed_fold (const float2* v, uint64_t span, uint64_t ndat, unsigned nchan,
                                unsigned npol, const FoldView& fv, cudaStream_t st,
                                const KernelClock* clk)
{
  if (ndat == 0) return cudaSuccess;
  const dim3 grid (unsigned ((ndat + 255) / 256), nchan);
  ClockScope cs (clk, KK_INV_COLS, st);
  if (fv.nout == 1)
    k_zeroed_fold<1><<<grid, 256, 0, st>>> (v, span, ndat, npol, fv);
  else if (fv.nout == 2)
    k_zeroed_fold<2><<<grid, 256, 0, st>>> (v, span, ndat, npol, fv);
  else
    k_zeroed_fold<4><<<grid, 256, 0, st>>> (v, span, ndat, npol, fv);
  return cudaGetLastError ();
}

cudaError_t launch_binplan (const FoldSegment* segs, int nseg, uint64_t ndat, unsigned nbin,
                            uint32_t* out, cudaStream_t st)
{
  if (ndat == 0) return cudaSuccess;
  g_launches++;
  k_binplan<<<unsigned ((ndat + 255) / 256), 256, 0, st>>> (segs, nseg, ndat, nbin, out);
  return cudaGetLastError ();
}

} // namespace b200
