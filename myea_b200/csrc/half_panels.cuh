// Operand panels of the dense contractions: an fp32 tensor as the sum of two half-precision arrays times powers of two.
//
//   x = (h0 + h1) * 2^e        h0 = x * 2^-e rounded to half, h1 = what is left of x * 2^-e rounded to half
//
// A contraction reads a tensor through its rows (K along the columns) or through its columns (K along the rows), and its
// results along the other index are independent of each other: a sample with huge inputs, a unit with tiny errors must not
// touch its neighbours.  So the exponent belongs to ONE row (column) and 128 of K, and a tensor that is read both ways has
// two sets, one per reading (4 bytes per element and set).  e puts the largest finite magnitude m of these 128 elements
// into [2^14, 2^15): an element of magnitude a is off by at most max(2^-22 a, 2^-39 m, 2^-127) - two halves carry 22 bits
// down to 2^-17 of m and then a fixed step.  Infinities and NaN stay what they are and reach the results of their own row and
// column only.  A product is h1_a*h0_b + h0_a*h1_b + h0_a*h0_b, three half instructions per 16 of K; the dropped h1_a*h1_b is
// 2^-22 of it.
// (With one exponent per block of 128 x 128 and one set for both readings an infinity turned every other row of its block
// into zeros, and rows or columns below 2^-22 of the block's largest lost digits that a TF32 + bf16 split keeps.  The second set
// costs 4 bytes written per element: activation of 4096 x 4096 47 -> 58 us, update of 138 M
// weights 699 -> 764 us, the training step around them 3 % longer.)
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace myea {

constexpr int HP_BLOCK = 128;   // rows and columns of a block with one exponent

// exponent for a row or column whose largest finite magnitude is amax; the scales 2^-e and 2^(e - 14) have to be normal floats
__device__ __forceinline__ int half_exponent(float amax) {
  const int E = static_cast<int>((__float_as_uint(amax) >> 23) & 0xFFu);
  if (amax == 0.f) return 0;
  return max(E - 127 - 14, -112);
}
// 2^n for -126 <= n <= 127
__device__ __forceinline__ float pow2(int n) { return __uint_as_float(static_cast<uint32_t>(n + 127) << 23); }

// the power of two as it is kept beside the panels: the upper half of the float 2^(e - 14) (see half_gemm.cu)
__device__ __forceinline__ uint16_t half_scale_bits(int e) { return static_cast<uint16_t>((e - 14 + 127) << 7); }

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
constexpr int HP_THREADS = 512;
constexpr int HP_ROWS = HP_BLOCK * 16 / HP_THREADS;   // rows per thread
__device__ __forceinline__ float finite_abs(float x) {
  x = fabsf(x);
  return x <= 3.402823466e+38f ? x : 0.f;
}
// largest finite magnitudes of a thread's rows and columns -> of the whole rows (16 lanes share them)
__device__ __forceinline__ void half_row_maxima(const float (&v)[HP_ROWS][8], float (&m)[HP_ROWS]) {
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    m[i] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) m[i] = fmaxf(m[i], finite_abs(v[i][j]));
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
  }
}
// ... and of the block's columns, over the 32 threads that share them (all threads of the block call it)
__device__ __forceinline__ void half_column_maxima(const float (&v)[HP_ROWS][8], float (&m)[8]) {
  __shared__ float4 part[HP_THREADS / 32][HP_BLOCK / 4];
  __shared__ float whole[HP_BLOCK];
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    m[j] = 0.f;
#pragma unroll
    for (int i = 0; i < HP_ROWS; ++i) m[j] = fmaxf(m[j], finite_abs(v[i][j]));
    m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], 16));
  }
  if (lane < 16) {
    part[threadIdx.x >> 5][2 * lane] = make_float4(m[0], m[1], m[2], m[3]);
    part[threadIdx.x >> 5][2 * lane + 1] = make_float4(m[4], m[5], m[6], m[7]);
  }
  __syncthreads();
  if (threadIdx.x < HP_BLOCK) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < HP_THREADS / 32; ++w) t = fmaxf(t, reinterpret_cast<const float *>(part[w])[threadIdx.x]);
    whole[threadIdx.x] = t;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = whole[(threadIdx.x & 15) * 8 + j];
}
// elements (r, c .. c + 7), already times 2^-e; c + 8 <= pitch, columns past the tensor's width are zeros
__device__ __forceinline__ void half_store8(const HalfPanels &p, const HalfReading &to, long long r, long long c, const float (&s)[8]) {
  uint4 h0, h1;
  half_split8(s, h0, h1);
  *reinterpret_cast<uint4 *>(to.h0 + r * p.pitch + c) = h0;
  *reinterpret_cast<uint4 *>(to.h1 + r * p.pitch + c) = h1;
}
// A block of the tensor, held by its 512 threads (zeros past the tensor's edges), into the panels of every reading that p has
__device__ __forceinline__ void half_store_block(const HalfPanels &p, long long by, long long bx, const float (&v)[HP_ROWS][8]) {
  const long long c = bx * HP_BLOCK + (threadIdx.x & 15) * 8, r0 = by * HP_BLOCK + (threadIdx.x >> 4);
  if (p.rows.h0 != nullptr) {
    float m[HP_ROWS];
    half_row_maxima(v, m);
#pragma unroll
    for (int i = 0; i < HP_ROWS; ++i) {
      const long long r = r0 + HP_THREADS / 16 * i;
      const int e = half_exponent(m[i]);
      if ((threadIdx.x & 15) == 0) p.rows.scale[bx * p.rows.pitch + r] = half_scale_bits(e);
      const float f = pow2(-e);
      float s[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = v[i][j] * f;
      if (r < p.R && c < p.pitch) half_store8(p, p.rows, r, c, s);
    }
  }
  if (p.cols.h0 != nullptr) {
    float m[8];
    half_column_maxima(v, m);
    uint32_t bits[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = half_exponent(m[j]);
      bits[j] = half_scale_bits(e);
      m[j] = pow2(-e);
    }
    if (threadIdx.x < 16)
      *reinterpret_cast<uint4 *>(p.cols.scale + by * p.cols.pitch + c) =
          make_uint4(bits[0] | bits[1] << 16, bits[2] | bits[3] << 16, bits[4] | bits[5] << 16, bits[6] | bits[7] << 16);
#pragma unroll
    for (int i = 0; i < HP_ROWS; ++i) {
      const long long r = r0 + HP_THREADS / 16 * i;
      float s[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = v[i][j] * m[j];
      if (r < p.R && c < p.pitch) half_store8(p, p.cols, r, c, s);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// A producer computes an fp32 tensor and leaves it both as an array and as panels for the contractions that read it next:
// one block of 128 x 128 per CTA, read once, the largest magnitudes of its rows and columns found on chip, everything written
// once.  Bound by HBM at 4096 x 4096 (34 us for the 201 MB of a split for both readings) and by the chain load - maximum - store
// of the one block an SM gets at 512 rows: 512 threads of 4 rows (activation of 512 x 4096 12.5 us).
// F: struct Cols; columns(Cols &, c, n): what belongs to this thread's columns c .. c + n - 1; row(cols, r, c, n, v): the
// values of row r (zeros in v[n] ..); keep(r, c, n, v): stores the fp32 result (may do nothing).
// ---------------------------------------------------------------------------------------------------------
// Eight values of which n are the tensor's (the others are zeros): as one access of 32 bytes where the address allows it, so that
// a warp asks for every sector once; two of 16 bytes each (vec: such addresses) ask twice, and their stores reach L2 as halves of
// sectors.  4096 x 4096: normalization backward 78 -> 74 us, activation 60 -> 57.
__device__ __forceinline__ bool whole_sector(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }
__device__ __forceinline__ void ld8(float (&d)[8], const float *p, int n, bool vec) {
  if (n == 8 && whole_sector(p)) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
                 : "l"(p) : "memory");
  } else if (vec && n == 8) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = j < n ? p[j] : 0.f;
  }
}
__device__ __forceinline__ void st8(float *p, const float (&d)[8], int n, bool vec) {
  if (n == 8 && whole_sector(p)) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(d[0]), "f"(d[1]), "f"(d[2]), "f"(d[3]), "f"(d[4]), "f"(d[5]),
                 "f"(d[6]), "f"(d[7]) : "memory");
  } else if (vec && n == 8) {
    *reinterpret_cast<float4 *>(p) = make_float4(d[0], d[1], d[2], d[3]);
    *reinterpret_cast<float4 *>(p + 4) = make_float4(d[4], d[5], d[6], d[7]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) p[j] = d[j];
  }
}

// block (by, bx) of the tensor: this thread's share of its values, zeros past the tensor's edges
template <typename F>
__device__ __forceinline__ void half_load_block(const F &f, long long R, long long C, long long by, long long bx, float (&v)[HP_ROWS][8]) {
  const long long c = bx * HP_BLOCK + (threadIdx.x & 15) * 8, r0 = by * HP_BLOCK + (threadIdx.x >> 4);
  const int n = static_cast<int>(max(0ll, min(8ll, C - c)));
  typename F::Cols cols;
  f.columns(cols, c, n);
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = r0 + HP_THREADS / 16 * i;
    if (r < R) {
      f.row(cols, r, c, n, v[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = r0 + HP_THREADS / 16 * i;
    if (r < R) f.keep(r, c, n, v[i]);
  }
}
__device__ __forceinline__ void half_block_of(long long C, unsigned block, unsigned &by, unsigned &bx) {
  // (one dimension: the row blocks of a tensor of many million rows are more than the others hold)
  const unsigned across = static_cast<unsigned>((C + HP_BLOCK - 1) / HP_BLOCK);
  by = block / across;
  bx = block - by * across;
}
inline unsigned half_blocks(long long R, long long C) { return static_cast<unsigned>(((C + HP_BLOCK - 1) / HP_BLOCK) * ((R + HP_BLOCK - 1) / HP_BLOCK)); }

template <typename F>
__global__ void __launch_bounds__(HP_THREADS, 2) half_produce_kernel(const F f, const HalfPanels p) {
  grid_dependency_wait();
  grid_dependency_release();
  unsigned by, bx;
  half_block_of(p.C, blockIdx.x, by, bx);
  float v[HP_ROWS][8];
  half_load_block(f, p.R, p.C, by, bx, v);
  half_store_block(p, by, bx, v);
}
template <typename F>
inline cudaError_t half_produce(const Context &ctx, const F &f, const HalfPanels &p) {
  return launch_dependent(ctx, half_produce_kernel<F>, dim3(half_blocks(p.R, p.C)), dim3(HP_THREADS), 0, f, p);
}

}  // namespace myea
