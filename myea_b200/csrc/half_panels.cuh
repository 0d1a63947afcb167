// Operand panels of the dense contractions: an fp32 tensor as the sum of two half-precision arrays times a power of two.
//
//   x = (h0 + h1) * 2^e        h0 = x * 2^-e rounded to half, h1 = what is left of x * 2^-e rounded to half
//
// Two halves carry 22 significant bits.  e is chosen per block of 128 x 128 elements so that the block's largest magnitude
// lands in [2^14, 2^15): an element of magnitude a in a block whose largest is m is off by at most max(2^-22 a, 2^-39 m) -
// half keeps 22 bits down to 2^-17 of the block's largest and then a fixed step of 2^-39 of it.  A product is
// h1_a*h0_b + h0_a*h1_b + h0_a*h0_b, three half instructions per 16 of K; the dropped h1_a*h1_b is 2^-22 of it.
// (Before: a TF32 array and, per reading, a bf16 cross-term array - 12 bytes per element for a tensor that is read through
// rows and columns, two instructions per 8 of K, products off by up to 2^-17.)  The same two arrays serve both operand
// roles and both readings, through their rows (K contiguous) and through their columns.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace myea {

constexpr int HP_BLOCK = 128;   // rows and columns of a block with one exponent

// exponent for a block whose largest magnitude is amax
__device__ __forceinline__ int half_exponent(float amax) {
  const int E = static_cast<int>((__float_as_uint(amax) >> 23) & 0xFFu);
  if (amax == 0.f) return 0;
  return max(E - 127 - 14, -126);   // (the scale 2^-e has to be a normal float)
}
// 2^n for -126 <= n <= 127
__device__ __forceinline__ float pow2(int n) { return __uint_as_float(static_cast<uint32_t>(n + 127) << 23); }

__device__ __forceinline__ uint32_t half2_bits(float a, float b) {   // a in the lower half
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float2 half2_floats(uint32_t h) { return __half22float2(*reinterpret_cast<const __half2 *>(&h)); }

// 8 consecutive elements (already times 2^-e) as 16 bytes of h0 and 16 bytes of h1
__device__ __forceinline__ void half_split8(const float (&v)[8], uint4 &h0, uint4 &h1) {
  uint32_t a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = half2_bits(v[2 * j], v[2 * j + 1]);
    const float2 f = half2_floats(a[j]);
    b[j] = half2_bits(v[2 * j] - f.x, v[2 * j + 1] - f.y);
  }
  h0 = make_uint4(a[0], a[1], a[2], a[3]);
  h1 = make_uint4(b[0], b[1], b[2], b[3]);
}

// A block of 512 threads holds a 128 x 128 block of the tensor: thread = 8 columns (tid % 16) of rows tid / 16 + 32 i.
// half_block_finish: the block's exponent from every thread's largest magnitude (all threads of the block call it).
constexpr int HP_THREADS = 512;
constexpr int HP_ROWS = HP_BLOCK * 16 / HP_THREADS;   // rows per thread
template <int THREADS = HP_THREADS>
__device__ __forceinline__ int half_block_exponent(float amax) {
  __shared__ float sh[THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = amax;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) amax = fmaxf(amax, sh[w]);
  return half_exponent(amax);
}
__device__ __forceinline__ float amax8(const float (&v)[8], float m) {
#pragma unroll
  for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(v[j]));
  return m;
}
// elements (r, c .. c + 7); c + 8 <= pitch, columns past the tensor's width are zeros
__device__ __forceinline__ void half_store8(const HalfPanels &p, long long r, long long c, const float (&v)[8], float scale) {
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = v[j] * scale;
  uint4 h0, h1;
  half_split8(s, h0, h1);
  *reinterpret_cast<uint4 *>(p.h0 + r * p.pitch + c) = h0;
  *reinterpret_cast<uint4 *>(p.h1 + r * p.pitch + c) = h1;
}

// ---------------------------------------------------------------------------------------------------------
// A producer computes an fp32 tensor and leaves it both as an array and as panels for the contractions that read it next:
// one block of 128 x 128 per CTA, read once, its largest magnitude found in registers, everything written once.  Bound by HBM
// at 4096 x 4096 (26 us for the 128 MB of a split) and by the chain load - maximum - store of the one block an SM gets at 512 rows:
// 512 threads of 4 rows (activation of 512 x 4096 11.3 us, with 256 threads of 8 rows 13.1).
// F: struct Cols; columns(Cols &, c, n): what belongs to this thread's columns c .. c + n - 1; row(cols, r, c, n, v): the
// values of row r (zeros in v[n] ..); keep(r, c, n, v): stores the fp32 result (may do nothing).
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ld8(float (&d)[8], const float *p, int n, bool vec) {
  if (vec && n == 8) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = j < n ? p[j] : 0.f;
  }
}
__device__ __forceinline__ void st8(float *p, const float (&d)[8], int n, bool vec) {
  if (vec && n == 8) {
    *reinterpret_cast<float4 *>(p) = make_float4(d[0], d[1], d[2], d[3]);
    *reinterpret_cast<float4 *>(p + 4) = make_float4(d[4], d[5], d[6], d[7]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) p[j] = d[j];
  }
}

template <typename F>
__global__ void __launch_bounds__(HP_THREADS, 2) half_produce_kernel(const F f, const HalfPanels p) {
  grid_dependency_wait();
  grid_dependency_release();
  // (one dimension: the row blocks of a tensor of many million rows are more than the others hold)
  const unsigned across = static_cast<unsigned>((p.C + HP_BLOCK - 1) / HP_BLOCK), by = blockIdx.x / across, bx = blockIdx.x - by * across;
  const long long c = bx * static_cast<long long>(HP_BLOCK) + (threadIdx.x & 15) * 8;
  const long long r0 = by * static_cast<long long>(HP_BLOCK) + (threadIdx.x >> 4);
  const int n = static_cast<int>(max(0ll, min(8ll, p.C - c)));
  typename F::Cols cols;
  f.columns(cols, c, n);
  float v[HP_ROWS][8], m = 0.f;
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = r0 + HP_THREADS / 16 * i;
    if (r < p.R) {
      f.row(cols, r, c, n, v[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) m = amax8(v[i], m);
  const int e = half_block_exponent(m);
  if (threadIdx.x == 0) p.exps[by * p.exp_r + bx * p.exp_c] = e;
  if (c >= p.pitch) return;
  const float scale = pow2(-e);
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = r0 + HP_THREADS / 16 * i;
    if (r >= p.R) continue;
    f.keep(r, c, n, v[i]);
    half_store8(p, r, c, v[i], scale);
  }
}
template <typename F>
inline cudaError_t half_produce(const Context &ctx, const F &f, const HalfPanels &p) {
  const dim3 grid(static_cast<unsigned>(((p.C + HP_BLOCK - 1) / HP_BLOCK) * ((p.R + HP_BLOCK - 1) / HP_BLOCK)));
  return launch_dependent(ctx, half_produce_kernel<F>, grid, dim3(HP_THREADS), 0, f, p);
}

}  // namespace myea
