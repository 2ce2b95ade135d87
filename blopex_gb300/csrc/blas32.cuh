// blas32.cuh -- building blocks of the FP32 column kernels (dot products and
// the inner-CG preconditioner's fused updates): 16-byte vector access and an
// FP32 accumulator that keeps FP64-level accuracy.
//
// On this GPU the FP64 pipe runs at 1/64 of the FP32 rate, so an FP32 dot
// product that accumulates in FP64 is bound by its DFMAs, not by HBM.  Here
// each product a b is made exact as p + e (e = fma(a, b, -p)) and added to a
// compensated FP32 sum (Knuth's two-sum); after at most 64 terms the pair (s, c)
// goes into an FP64 accumulator or, first, is merged with other threads' pairs.  The intrinsics keep the compiler from
// contracting the two-sum into FMAs, which would break its error term.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

static __device__ __forceinline__ void acc_prod32(float& s, float& c, float a, float b)
{
  const float p = __fmul_rn(a, b);
  const float e = fmaf(a, b, -p);  // a b = p + e exactly (no underflow)
  const float t = __fadd_rn(s, p);
  const float bp = __fsub_rn(t, s);
  const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
  c = __fadd_rn(c, __fadd_rn(err, e));
  s = t;
}

static __device__ __forceinline__ void acc_prod32x4(float& s, float& c, float4 a, float4 b)
{
  acc_prod32(s, c, a.x, b.x);
  acc_prod32(s, c, a.y, b.y);
  acc_prod32(s, c, a.z, b.z);
  acc_prod32(s, c, a.w, b.w);
}

// (s, c) += (s2, c2), two compensated sums
static __device__ __forceinline__ void acc_pair32(float& s, float& c, float s2, float c2)
{
  const float t = __fadd_rn(s, s2);
  const float bp = __fsub_rn(t, s);
  const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(s2, bp));
  s = t;
  c = __fadd_rn(__fadd_rn(c, c2), e);
}

static __device__ __forceinline__ void two_sum32(float& s, float& e, float a, float b)
{
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// (s, c, d) += (s2, c2, d2): the roundings of the second word kept in a third, for
// long merges of compensated sums
static __device__ __forceinline__ void acc_triple32(float& s, float& c, float& d, float s2, float c2, float d2)
{
  float t, e, u, g, v, h;
  two_sum32(t, e, s, s2);
  two_sum32(u, g, c, c2);
  two_sum32(v, h, u, e);
  s = t;
  c = v;
  d = __fadd_rn(__fadd_rn(d, d2), __fadd_rn(g, h));
}

static __device__ __forceinline__ void warp_pair_sum32(float& s, float& c)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o), c2 = __shfl_xor_sync(0xffffffffu, c, o);
    acc_pair32(s, c, s2, c2);
  }
}

// block-wide sum of the threads' compensated sums (blockDim.x = 256), the
// result in thread 0, in a fixed order: the warps in FP32 pairs (an FP64 add
// holds this GPU's FP64 pipe for 16 cycles), the eight warp sums in FP64
static __device__ __forceinline__ double block_pair_sum256(float s, float c)
{
  __shared__ float2 red[8];
  warp_pair_sum32(s, c);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(s, c);
  __syncthreads();
  double v = 0.0;
  if (threadIdx.x < 32) {
    const float2 p = red[threadIdx.x & 7];
    v = (double)p.x + (double)p.y;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  return v;
}

// block-wide sum of one double per thread (blockDim.x = 256), the result in
// thread 0, in a fixed order: halves of 128, 64, ..., 1.  All of it in warp 0
// behind one branch: a tree over the block, its adds predicated off in the warps
// that had no part in a level, held the FP64 pipe (16 cycles an instruction,
// executed or not) for 1024 cycles a block instead of 192.
static __device__ __forceinline__ double block_sum256(double v)
{
  __shared__ double red[256];
  const int t = threadIdx.x;
  red[t] = v;
  __syncthreads();
  if (t < 32) {
    const double a0 = red[t] + red[t + 128], a1 = red[t + 32] + red[t + 160];
    const double a2 = red[t + 64] + red[t + 192], a3 = red[t + 96] + red[t + 224];
    v = (a0 + a2) + (a1 + a3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// p[0] + p[1] + ... + p[n - 1] in that order, in thread 0 (blockDim.x = 256): the
// loads by the whole block at once, the adds one by one (70 cycles each)
static __device__ __forceinline__ double ordered_sum256(const double* p, int n)
{
  __shared__ double buf[256];
  double s = 0.0;
  for (int b0 = 0; b0 < n; b0 += 256) {
    if (b0 + threadIdx.x < n) buf[threadIdx.x] = __ldcg(p + b0 + threadIdx.x);
    __syncthreads();
    if (threadIdx.x == 0) {
      const int m = min(256, n - b0);
#pragma unroll 8
      for (int b = 0; b < m; b++) s += buf[b];
    }
    __syncthreads();
  }
  return s;
}

static inline bool cols_aligned16(const void* const* cols, int w)
{
  for (int j = 0; j < w; j++)
    if ((uintptr_t)cols[j] & 15) return false;
  return true;
}
