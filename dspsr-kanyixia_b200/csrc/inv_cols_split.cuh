// inv_cols_split.cuh -- inverse column pass, two polarisations, a thread per
// polarisation (and half column)
#pragma once

#include "device_common.cuh"
#include "dft_pair.cuh"

namespace b200 {

namespace {

// What the inverse column pass of the convolution and of the filterbank with a
// response share: columns of n1 values n2 apart; column i2 is sample
// t2 = i2 mod seg of channel cin * (n2 / seg) + i2 / seg, value k after the
// transform is sample k * seg + t2 of the part (the convolution: seg = n2).
struct InvColsShape
{
  unsigned n2, seg, nchan_in;
  uint64_t nkeep;
  unsigned nfilt_pos;
};

// threads per column: two polarisations, and at n1 = 32 two halves each
template <int N1> B200_CE int ivs_split () { return N1 == 32 ? 4 : 2; }
template <int N1> B200_CE int ivs_cols () { return 128 / ivs_split<N1> (); }
// resident blocks per SM that the registers are sized for
template <int N1> B200_CE int ivs_blocks () { return N1 == 8 ? 10 : 8; }

// K3 with detection and fold, for two polarisations and n1 = 8, 16 or 32.  A
// thread transforms one polarisation of one column (at n1 = 32 the even or the
// odd rows of it), so that it needs 64 registers or less and 32 warps and more
// keep loads in flight: the pass waits for HBM and for the latency of the fold's shuffles,
// and a thread per column with both polarisations (128 to 168 registers, 11
// to 16 warps per SM) left 60 % of the issue slots empty.  The values are
// exchanged through shared memory, after which every thread has both
// polarisations of n1 / 2 (8, 16) or eight (32) of the column's samples; the
// last radix-2 step of n1 = 32 is taken there.  The twiddles of the block's
// columns stay in shared memory for all its parts (b = blockIdx.y,
// + gridDim.y, ...).  A thread per column and now: 239 and 162 us at n1 = 16
// (10.5 M samples of one channel, long bins; 192 us at n1 = 32, where 2^17
// points go with 4096-point rows), 174 and 99 us at n1 = 32 (2^18 points), and
// for the filterbank with a response (n1 = 32) 615 and 363 us.
template <int N1, int NOUT, bool LONG>
__global__ void __launch_bounds__ (128, ivs_blocks<N1> ())
k_inv_cols_split (const float2* __restrict__ scratch, const InvColsShape sh, const uint64_t part0,
                  const unsigned nbatch, const float2* __restrict__ tw, const FoldView fv)
{
  constexpr int HS = N1 == 32 ? 2 : 1;            // halves of a column
  constexpr int V = N1 / HS;                      // values per thread
  constexpr int COLS = ivs_cols<N1> ();
  // n1 = 32: [pol][half][j][col]; otherwise the values handed over, [pol][m][col]
  __shared__ __align__ (16) float2 s_x[(HS == 2 ? 2 : 1) * N1 * COLS];
  __shared__ float2 s_tw[N1 * COLS];                     // [k][col]
  using RF = RowFold<NOUT, NOUT == 4 || N1 == 8 ? 4 : 8>;
  __shared__ __align__ (16) float s_fold[LONG ? 4 * RF::WORDS : 4];
  const unsigned col = threadIdx.x % COLS, part_of = threadIdx.x / COLS;
  const unsigned pol = part_of & 1, h = part_of >> 1;
  const unsigned i0 = blockIdx.x * COLS, i2 = i0 + col;
  const unsigned cin = blockIdx.z, c = cin * (sh.n2 / sh.seg) + i0 / sh.seg;
  const unsigned t2 = i2 % sh.seg;
  const uint64_t N = uint64_t (N1) * sh.n2;
  RF rf (s_fold + (LONG ? (threadIdx.x >> 5) * RF::WORDS : 0),
         fv.profiles + uint64_t (c) * NOUT * fv.stride, fv.stride, c == 0 ? fv.hits : nullptr);
  for (unsigned e = threadIdx.x; e < unsigned (N1 * COLS); e += 128)
    s_tw[e] = __ldg (tw + uint64_t (e / COLS) * sh.seg + i0 % sh.seg + e % COLS);
  constexpr int R = N1 == 32 ? 8 : N1 / 2;        // samples the thread detects
  // sample r of the thread after the exchange
  const auto sample = [&] (int r) {
    return HS == 2 ? 4 * (r >> 1) + int (part_of) + 16 * (r & 1) : 2 * r + int (pol);
  };
  for (unsigned b = blockIdx.y; b < nbatch; b += gridDim.y)
  {
    const uint64_t tbase = (part0 + b) * sh.nkeep;
    const float2* src = scratch + ((uint64_t (b) * sh.nchan_in + cin) * 2 + pol) * N + i2;
    float2 v[V];
#pragma unroll
    for (int m = 0; m < V; m++) v[m] = __ldcs (src + uint64_t (HS * m + h) * sh.n2);
    // the profile columns of the samples, asked for with the values: waited for
    // one after another in the fold they were most of the pass's time
    unsigned fcol[R];
#pragma unroll
    for (int r = 0; r < R; r++)
    {
      const uint64_t tl = uint64_t (sample (r)) * sh.seg + t2;
      const bool ok = tl >= sh.nfilt_pos && tl < sh.nfilt_pos + sh.nkeep;
      fcol[r] = fold_column (fv, ok, tbase + (tl - sh.nfilt_pos));
    }
    __syncthreads ();                  // the twiddles are there; the last part's reads are done
#pragma unroll
    for (int m = 0; m < V; m++)
      if (HS == 2 || m) v[m] = cmulc (v[m], s_tw[(HS * m + h) * COLS + col]);
    dft::run<V, +1> (v);
    // n1 = 32: X[j] and X[j + 16] are E[j] +- w32^j O[j]
    if (HS == 2 && h)
    {
#pragma unroll
      for (int j = 1; j < V; j++) v[j] = dft::tw64<+1> (2 * j, v[j]);
    }
    if constexpr (HS == 2)
    {
      float2* x = s_x + (pol * N1 + h * V) * COLS + col;
#pragma unroll
      for (int j = 0; j < V; j++) x[j * COLS] = v[j];
    }
    else
    {
      // the thread of polarisation 0 keeps the even samples and hands over the
      // odd ones, the other the reverse
      float2* x = s_x + pol * (N1 / 2) * COLS + col;
#pragma unroll
      for (int m = 0; m < N1 / 2; m++)
      {
        x[m * COLS] = pol ? v[2 * m] : v[2 * m + 1];
        v[m] = pol ? v[2 * m + 1] : v[2 * m];
      }
    }
    __syncthreads ();
    const auto emit = [&] (int r, float2 p, float2 q) {
      detect_row<LONG> (rf, fv.state, 2, fcol[r], p, q);
      if (LONG && (r + 1) % RF::ROWS == 0) rf.flush ();
    };
    if constexpr (HS == 1)
    {
      const float2* y = s_x + (pol ^ 1) * (N1 / 2) * COLS + col;
#pragma unroll
      for (int r = 0; r < R; r++)
      {
        const float2 z = y[r * COLS];
        emit (r, pol ? z : v[r], pol ? v[r] : z);
      }
    }
    else
    {
      const float2* y = s_x + col;
#pragma unroll
      for (int m = 0; m < 4; m++)
      {
        const int j = 4 * m + int (part_of);
        const float2 ep = y[j * COLS], op = y[(16 + j) * COLS];
        const float2 eq = y[(32 + j) * COLS], oq = y[(48 + j) * COLS];
        emit (2 * m, cadd (ep, op), cadd (eq, oq));
        emit (2 * m + 1, csub (ep, op), csub (eq, oq));
      }
    }
  }
}

template <int N1, int NOUT>
void launch_inv_split (const float2* scratch, const InvColsShape& sh, uint64_t part0,
                       unsigned nbatch, const float2* tw, int nsm, const FoldView& fv,
                       cudaStream_t st)
{
  const unsigned gx = sh.n2 / ivs_cols<N1> ();
  // about four blocks of work per resident block, then parts per block
  const unsigned resident = unsigned (nsm) * ivs_blocks<N1> ();
  const unsigned want = std::max (1u, 4 * resident / std::max (1u, gx * sh.nchan_in));
  const dim3 grid (gx, std::min (nbatch, want), sh.nchan_in);
  if (fv.long_bins)
    k_inv_cols_split<N1, NOUT, true><<<grid, 128, 0, st>>> (scratch, sh, part0, nbatch, tw, fv);
  else
    k_inv_cols_split<N1, NOUT, false><<<grid, 128, 0, st>>> (scratch, sh, part0, nbatch, tw, fv);
}

} // namespace

} // namespace b200
