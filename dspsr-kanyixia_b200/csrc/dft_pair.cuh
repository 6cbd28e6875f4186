// dft_pair.cuh -- in-register DFTs of one complex value or of both
// polarisations at once.
//
// C2 holds the two polarisations of one sample as (re0, re1), (im0, im1):
// every add, multiply and fma of a transform then works on both through one
// fma.rn.f32x2-class instruction, with the rounding of the scalar form.  The
// FP32 pipes run at the same rate either way (128 lanes per clock and SM), but
// a transform takes half the issue slots and each twiddle serves both
// polarisations.  (Packing re with im instead needs register moves for every
// twiddle and for i z: it measured slower in every column kernel.)
#pragma once

#include "fft_core.cuh"

namespace b200 {

struct C2
{
  float2 re, im;
};

// One complex value whose adds are packed (re with im): the packed form saves
// issue slots wherever no operand has to be rearranged; twiddle products and
// +- i stay scalar.
struct CP
{
  float2 z;
};

#ifdef __CUDACC__

namespace dft {

__device__ __forceinline__ float2 dup (float a) { return make_float2 (a, a); }

__device__ __forceinline__ float2 add (float2 a, float2 b) { return cadd (a, b); }
__device__ __forceinline__ float2 sub (float2 a, float2 b) { return csub (a, b); }
// a + i b, a - i b
__device__ __forceinline__ float2 addi (float2 a, float2 b) { return make_float2 (a.x - b.y, a.y + b.x); }
__device__ __forceinline__ float2 subi (float2 a, float2 b) { return make_float2 (a.x + b.y, a.y - b.x); }
// a * (c + i s)
__device__ __forceinline__ float2 mulc (float2 a, float c, float s)
{
  return make_float2 (a.x * c - a.y * s, a.x * s + a.y * c);
}
// a + h b
__device__ __forceinline__ float2 fmah (float2 a, float h, float2 b)
{
  return make_float2 (fmaf (h, b.x, a.x), fmaf (h, b.y, a.y));
}

// a - b without a negated operand: fma with -1 rounds as the subtraction
__device__ __forceinline__ float2 sub2 (float2 a, float2 b) { return __ffma2_rn (b, dup (-1.f), a); }
__device__ __forceinline__ C2 add (C2 a, C2 b)
{
  return {__fadd2_rn (a.re, b.re), __fadd2_rn (a.im, b.im)};
}
__device__ __forceinline__ C2 sub (C2 a, C2 b) { return {sub2 (a.re, b.re), sub2 (a.im, b.im)}; }
__device__ __forceinline__ C2 addi (C2 a, C2 b) { return {sub2 (a.re, b.im), __fadd2_rn (a.im, b.re)}; }
__device__ __forceinline__ C2 subi (C2 a, C2 b) { return {__fadd2_rn (a.re, b.im), sub2 (a.im, b.re)}; }
__device__ __forceinline__ C2 mulc (C2 a, float c, float s)
{
  return {__ffma2_rn (a.re, dup (c), __fmul2_rn (a.im, dup (-s))),
          __ffma2_rn (a.re, dup (s), __fmul2_rn (a.im, dup (c)))};
}
__device__ __forceinline__ C2 fmah (C2 a, float h, C2 b)
{
  return {__ffma2_rn (b.re, dup (h), a.re), __ffma2_rn (b.im, dup (h), a.im)};
}

__device__ __forceinline__ CP add (CP a, CP b) { return {__fadd2_rn (a.z, b.z)}; }
__device__ __forceinline__ CP sub (CP a, CP b) { return {sub2 (a.z, b.z)}; }
__device__ __forceinline__ CP addi (CP a, CP b) { return {addi (a.z, b.z)}; }
__device__ __forceinline__ CP subi (CP a, CP b) { return {subi (a.z, b.z)}; }
__device__ __forceinline__ CP mulc (CP a, float c, float s) { return {mulc (a.z, c, s)}; }
__device__ __forceinline__ CP fmah (CP a, float h, CP b) { return {__ffma2_rn (b.z, dup (h), a.z)}; }

// a + D i b
template <int D, typename T> __device__ __forceinline__ T addj (T a, T b)
{
  return D > 0 ? addi (a, b) : subi (a, b);
}

// D i v
template <int D> __device__ __forceinline__ float2 muli (float2 v)
{
  return D > 0 ? make_float2 (-v.y, v.x) : make_float2 (v.y, -v.x);
}
template <int D> __device__ __forceinline__ CP muli (CP v) { return {muli<D> (v.z)}; }
template <int D> __device__ __forceinline__ C2 muli (C2 v)
{
  return D > 0 ? C2 {__fmul2_rn (v.im, dup (-1.f)), v.re} : C2 {v.im, __fmul2_rn (v.re, dup (-1.f))};
}

// v * exp(D 2 pi i j / 64), j a compile-time constant after unrolling
template <int D, typename T> __device__ __forceinline__ T tw64 (int j, T v)
{
  if (j == 16) return muli<D> (v);
  const float c = cos64 (j), s = D < 0 ? -sin64 (j) : sin64 (j);
  return mulc (v, c, s);
}

template <int D, typename T> __device__ __forceinline__ void dft4 (T& a, T& b, T& c, T& d)
{
  const T s = add (a, c), t = sub (a, c), u = add (b, d), w = sub (b, d);
  a = add (s, u);
  c = sub (s, u);
  b = addj<D> (t, w);
  d = addj<-D> (t, w);
}

// natural order in and out; the sqrt(1/2) of the odd outputs rides in the
// final adds as fma
template <int D, typename T> __device__ __forceinline__ void dft8 (T* v)
{
  T e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  T o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<D> (e0, e1, e2, e3);
  dft4<D> (o0, o1, o2, o3);
  const float h = quarter_cos64 (8);
  const T r1 = addj<D> (o1, o1);          // (1 + D i) o1
  const T r3 = addj<-D> (o3, o3);         // (1 - D i) o3; w8^3 = -h (1 - D i)
  v[0] = add (e0, o0);
  v[4] = sub (e0, o0);
  v[1] = fmah (e1, h, r1);
  v[5] = fmah (e1, -h, r1);
  v[2] = addj<D> (e2, o2);
  v[6] = addj<-D> (e2, o2);
  v[3] = fmah (e3, -h, r3);
  v[7] = fmah (e3, h, r3);
}

// N-point DFT in place, natural order in and out, N = 2 .. 32
template <int N, int D, typename T> __device__ __forceinline__ void run (T* v)
{
  if constexpr (N == 2)
  {
    const T a = v[0], b = v[1];
    v[0] = add (a, b);
    v[1] = sub (a, b);
  }
  else if constexpr (N == 4)
    dft4<D> (v[0], v[1], v[2], v[3]);
  else if constexpr (N == 8)
    dft8<D> (v);
  else
  {
    // N = 4 x M: X[k1 + 4 k2] = sum_n2 w_M^(n2 k2) w_N^(n2 k1)
    // sum_n1 x[M n1 + n2] w_A^(n1 k1)
    constexpr int A = 4, M = N / A;
    T u[N];
#pragma unroll
    for (int n2 = 0; n2 < M; n2++)
    {
      T a = v[n2], b = v[M + n2], c = v[2 * M + n2], d = v[3 * M + n2];
      dft4<D> (a, b, c, d);
      u[n2] = a;
      u[M + n2] = n2 ? tw64<D> (n2 * 64 / N, b) : b;
      u[2 * M + n2] = n2 ? tw64<D> (2 * n2 * 64 / N, c) : c;
      u[3 * M + n2] = n2 ? tw64<D> (3 * n2 * 64 / N, d) : d;
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++)
    {
      run<M, D> (u + M * k1);
#pragma unroll
      for (int k2 = 0; k2 < M; k2++) v[k1 + A * k2] = u[M * k1 + k2];
    }
  }
}

} // namespace dft

#endif // __CUDACC__

} // namespace b200
