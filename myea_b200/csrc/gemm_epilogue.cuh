// The fused epilogue of the contraction kernels: what happens to a block of the product between the accumulators and
// global memory (bias, skip-connection addend, activation derivative with the normalization folded in, accumulation,
// column statistics), warp-collective over 32 x 32 blocks and element-wise for kernels that hold single elements.
#pragma once

#include "common.cuh"

namespace myea {

// epilogue math for one element
// offset of output row m from e.C: plain pitch, or one of up to four row segments that start at their own offsets
__device__ __forceinline__ long long c_row(const Epilogue &e, long long m) {
  if (e.seg_rows == 0) return m * e.ldc;
  const int s = static_cast<int>(m >= e.seg_rows) + static_cast<int>(m >= 2 * e.seg_rows) + static_cast<int>(m >= 3 * e.seg_rows);
  return (m - s * e.seg_rows) * e.ldc + e.seg_off[s];
}

// The derivative switch has two dozen cases.  In the element-wise epilogue the functions networks are made of are inline
// and the others go through one call; the unrolled block epilogues carry the inline ones only (derivative_is_fused).
static __device__ __noinline__ float af_derive_rare(uint32_t af, float z, float y) { return af_derive(af, z, y); }
template <bool RARE>
__device__ __forceinline__ float af_derive_common(uint32_t af, float z, float y) {
  switch (af) {
    case MYEA_AF_TANH: return af_derive(MYEA_AF_TANH, z, y);
    case MYEA_AF_SIGMOID: return af_derive(MYEA_AF_SIGMOID, z, y);
    case MYEA_AF_RELU: return af_derive(MYEA_AF_RELU, z, y);
    case MYEA_AF_LEAKY_RELU: return af_derive(MYEA_AF_LEAKY_RELU, z, y);
    case MYEA_AF_ELU: return af_derive(MYEA_AF_ELU, z, y);
    case MYEA_AF_SELU: return af_derive(MYEA_AF_SELU, z, y);
    case MYEA_AF_LINEAR: case MYEA_AF_LINEAR_PIECE: case MYEA_AF_LINEAR_PIECE_SYMMETRIC: case MYEA_AF_SOFTMAX: return 1.0f;
    default: return RARE ? af_derive_rare(af, z, y) : 1.0f;
  }
}

// RARE: whether the rarely used functions may occur
template <bool RARE = true>
__device__ __forceinline__ float epilogue_value(const Epilogue &e, float acc, long long m, long long n) {
  float v = acc;
  if (e.bias != nullptr) v += e.bias[n];
  if (e.addend != nullptr) v += e.addend[m * e.ld_addend + n];
  if (e.deriv_af != 0u) {
    float pre = 0.f, y = 0.f;
    if (e.aux_pre != nullptr) {
      pre = e.aux_pre[m * e.ld_aux + n];
      if (e.col_scale != nullptr) pre = pre * e.col_scale[n] + e.col_shift[n];
    }
    if (e.aux_y != nullptr) y = e.aux_y[m * e.ld_aux + n];
    v *= af_derive_common<RARE>(e.deriv_af, pre, y);
  }
  if (e.accumulate) v += e.C[c_row(e, m) + n];
  return v;
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// The vector path of the epilogue needs 16-byte aligned bases and pitches that are multiples of four floats.
__device__ __forceinline__ bool epilogue_vector_ok(const Epilogue &e) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(e.C) | reinterpret_cast<uintptr_t>(e.bias) | reinterpret_cast<uintptr_t>(e.addend) |
                         reinterpret_cast<uintptr_t>(e.aux_pre) | reinterpret_cast<uintptr_t>(e.aux_y) |
                         reinterpret_cast<uintptr_t>(e.col_scale) | reinterpret_cast<uintptr_t>(e.col_shift);
  return (bits & 15) == 0 && ((e.ldc | e.ld_addend | e.ld_aux | e.seg_off[0] | e.seg_off[1] | e.seg_off[2] | e.seg_off[3]) & 3) == 0;
}
// 0 plain (bias only), 1 activation derivative, 2 accumulate, 3 anything else
__device__ __forceinline__ int epilogue_mode(const Epilogue &e) {
  if (e.addend != nullptr) return 3;
  if (e.deriv_af != 0u) return e.accumulate ? 3 : 1;
  return e.accumulate ? 2 : 0;
}

// Epilogue of a 32-row x 32-column block, warp-collective: lane l holds row row0 + l (that is how tensor memory hands an
// accumulator to a warp), but global memory wants rows of 128 contiguous bytes.  The block goes through a 16 x 36
// float staging buffer in shared memory, half at a time: the owning lanes write their rows as float4 (conflict-free at
// pitch 36), then every lane takes one float4 column slot (lane % 8) of the rows lane / 8 + 4 i, so that each global
// instruction of the warp covers four full 128-byte row segments.  The loads of the four rows are issued before their
// first use.  ADD / DERIV / ACC say what MAY be present.  `tr`: this warp's 16 * 36 floats.
constexpr int TR_PITCH = 36;
constexpr int TR_WARP_FLOATS = 16 * TR_PITCH;

// x[i] *= f'(z[i], y[i]) for four float4; the activation is the same for the whole launch, so the switch is taken once
// per call and every case is straight-line code (a switch per element made this epilogue as long as a whole tile's
// main loop)
template <uint32_t AF>
__device__ __forceinline__ void derive4x4(float4 (&x)[4], const float4 (&z)[4], const float4 (&y)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i].x *= af_derive(AF, z[i].x, y[i].x);
    x[i].y *= af_derive(AF, z[i].y, y[i].y);
    x[i].z *= af_derive(AF, z[i].z, y[i].z);
    x[i].w *= af_derive(AF, z[i].w, y[i].w);
  }
}
__device__ __forceinline__ void derive4x4_any(uint32_t af, float4 (&x)[4], const float4 (&z)[4], const float4 (&y)[4]) {
  switch (af) {
    case MYEA_AF_TANH: derive4x4<MYEA_AF_TANH>(x, z, y); break;
    case MYEA_AF_SIGMOID: derive4x4<MYEA_AF_SIGMOID>(x, z, y); break;
    case MYEA_AF_RELU: derive4x4<MYEA_AF_RELU>(x, z, y); break;
    case MYEA_AF_LEAKY_RELU: derive4x4<MYEA_AF_LEAKY_RELU>(x, z, y); break;
    case MYEA_AF_ELU: derive4x4<MYEA_AF_ELU>(x, z, y); break;
    case MYEA_AF_SELU: derive4x4<MYEA_AF_SELU>(x, z, y); break;
    case MYEA_AF_LINEAR: case MYEA_AF_LINEAR_PIECE: case MYEA_AF_LINEAR_PIECE_SYMMETRIC: case MYEA_AF_SOFTMAX: break;  // derivative 1
    default: break;  // gemm_panels applies the rarely used functions in a pass of its own (derivative_is_fused)
  }
}

template <bool ADD, bool DERIV, bool ACC, int STATS = 0>
__device__ __forceinline__ void epilogue_block32(const Epilogue &e, float *tr, const float (&v)[32], int lane, long long row0, long long col0, int M) {
  const int c4 = (lane & 7) * 4, rsub = lane >> 3;
  const long long n = col0 + c4;
  const bool has_add = ADD && e.addend != nullptr, has_pre = DERIV && e.aux_pre != nullptr, has_y = DERIV && e.aux_y != nullptr;
  const bool affine = has_pre && e.col_scale != nullptr;
  const bool acc = ACC && e.accumulate;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 bias = e.bias != nullptr ? ld4(e.bias + n) : zero;
  const float4 cs = affine ? ld4(e.col_scale + n) : make_float4(1.f, 1.f, 1.f, 1.f), ch = affine ? ld4(e.col_shift + n) : zero;
  // The global reads of BOTH halves go out before anything else (one memory round trip per block instead of two);
  // the variant that may read all four arrays keeps to one half at a time for the sake of registers.
  constexpr bool AHEAD = !(ADD && DERIV && ACC);
  constexpr int SLOTS = AHEAD ? 8 : 4;
  float4 add[ADD ? SLOTS : 1], pre[DERIV ? SLOTS : 1], y[DERIV ? SLOTS : 1], old[ACC ? SLOTS : 1];
  auto load_rows = [&](int first_slot, int h0, int h1) {
#pragma unroll
    for (int h = h0; h < h1; ++h) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = first_slot + (h - h0) * 4 + i;
        const long long m = row0 + h * 16 + rsub + 4 * i;
        const bool in = m < M;
        if (ADD) add[s] = (has_add && in) ? ld4(e.addend + m * e.ld_addend + n) : zero;
        if (DERIV) {
          pre[s] = (has_pre && in) ? ld4(e.aux_pre + m * e.ld_aux + n) : zero;
          y[s] = (has_y && in) ? ld4(e.aux_y + m * e.ld_aux + n) : zero;
        }
        if (ACC) old[s] = (acc && in) ? ld4(e.C + c_row(e, m) + n) : zero;
      }
    }
  };
  // column statistics of this 32 x 32 block: this lane's four columns over its eight rows first
  float4 st0 = zero, st1 = zero;
  const float4 mu = (STATS == 2 && e.col_mean != nullptr) ? ld4(e.col_mean + n) : zero;
  if (AHEAD) load_rows(0, 0, 2);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!AHEAD) load_rows(0, h, h + 1);
    const int s0 = AHEAD ? h * 4 : 0;
    __syncwarp();
    if ((lane >> 4) == h) {
      float *dst = tr + (lane & 15) * TR_PITCH;
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(dst + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    __syncwarp();
    float4 x[4], z4[4], y4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = *reinterpret_cast<const float4 *>(tr + (rsub + 4 * i) * TR_PITCH + c4);
      x[i].x += bias.x; x[i].y += bias.y; x[i].z += bias.z; x[i].w += bias.w;
      if (ADD) { x[i].x += add[s0 + i].x; x[i].y += add[s0 + i].y; x[i].z += add[s0 + i].z; x[i].w += add[s0 + i].w; }
      if (DERIV) {
        const float4 p = pre[s0 + i];
        z4[i] = make_float4(p.x * cs.x + ch.x, p.y * cs.y + ch.y, p.z * cs.z + ch.z, p.w * cs.w + ch.w);
        y4[i] = y[s0 + i];
      }
    }
    if (DERIV) derive4x4_any(e.deriv_af, x, z4, y4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long m = row0 + h * 16 + rsub + 4 * i;
      if (ACC) { x[i].x += old[s0 + i].x; x[i].y += old[s0 + i].y; x[i].z += old[s0 + i].z; x[i].w += old[s0 + i].w; }
      if (m < M) {
        *reinterpret_cast<float4 *>(e.C + c_row(e, m) + n) = x[i];
        if (STATS == 1) {
          st0.x += x[i].x; st0.y += x[i].y; st0.z += x[i].z; st0.w += x[i].w;
          st1.x = fmaf(x[i].x, x[i].x, st1.x); st1.y = fmaf(x[i].y, x[i].y, st1.y); st1.z = fmaf(x[i].z, x[i].z, st1.z); st1.w = fmaf(x[i].w, x[i].w, st1.w);
        }
        if (STATS == 2) {
          const float4 p = pre[s0 + i];  // the raw array the derivative was taken on (before the folded normalization)
          st0.x += x[i].x; st0.y += x[i].y; st0.z += x[i].z; st0.w += x[i].w;
          st1.x = fmaf(x[i].x, p.x - mu.x, st1.x); st1.y = fmaf(x[i].y, p.y - mu.y, st1.y); st1.z = fmaf(x[i].z, p.z - mu.z, st1.z); st1.w = fmaf(x[i].w, p.w - mu.w, st1.w);
        }
      }
    }
  }
  if (STATS != 0) {
    // the four lanes that share a column slot (lane, lane ^ 8, lane ^ 16, lane ^ 24) hold the block's 32 rows between them
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
      st0.x += __shfl_xor_sync(0xffffffffu, st0.x, o); st0.y += __shfl_xor_sync(0xffffffffu, st0.y, o);
      st0.z += __shfl_xor_sync(0xffffffffu, st0.z, o); st0.w += __shfl_xor_sync(0xffffffffu, st0.w, o);
      st1.x += __shfl_xor_sync(0xffffffffu, st1.x, o); st1.y += __shfl_xor_sync(0xffffffffu, st1.y, o);
      st1.z += __shfl_xor_sync(0xffffffffu, st1.z, o); st1.w += __shfl_xor_sync(0xffffffffu, st1.w, o);
    }
    const long long blk = row0 >> 5;
    if (lane < 8 && blk < e.stats_blocks) {
      float *dst = e.col_stats + blk * e.ldc + n;   // [block][N]: the result's pitch is N for the arrays that ask for this
      *reinterpret_cast<float4 *>(dst) = st0;
      *reinterpret_cast<float4 *>(dst + e.stats_blocks * e.ldc) = st1;
    }
  }
}

// The same block for arrays the vector path cannot take (bases or pitches that are not multiples of 16 bytes: the weight
// derivatives of LSTM layers land inside the reference's per-block parameter layout, whose row pitch is odd) and for the
// ragged right edge: staged through the same buffer, then lane l takes column col0 + l of one row after the other, so a
// warp's accesses still cover one contiguous row segment each.
__device__ __forceinline__ void epilogue_block32_rows(const Epilogue &e, float *tr, const float (&v)[32], int lane, long long row0, long long col0, int M, int N) {
  const long long n = col0 + lane;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    __syncwarp();
    if ((lane >> 4) == h) {
      float *dst = tr + (lane & 15) * TR_PITCH;
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(dst + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    __syncwarp();
    if (e.accumulate && e.bias == nullptr && e.addend == nullptr && e.deriv_af == 0u) {
      // C += product and nothing else (weight derivatives): the 16 old row segments are requested together - one after
      // the other, their latency (rows of an LSTM layer's weight derivatives lie a whole block apart) is what the
      // epilogue of a tile takes
      float old[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const long long m = row0 + h * 16 + r;
        old[r] = (m < M && n < N) ? e.C[c_row(e, m) + n] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const long long m = row0 + h * 16 + r;
        if (m < M && n < N) e.C[c_row(e, m) + n] = tr[r * TR_PITCH + lane] + old[r];
      }
    } else {
#pragma unroll 4
      for (int r = 0; r < 16; ++r) {
        const long long m = row0 + h * 16 + r;
        if (m < M && n < N) e.C[c_row(e, m) + n] = epilogue_value<false>(e, tr[r * TR_PITCH + lane], m, n);
      }
    }
  }
}

// Warp-collective: every lane of the warp calls it (row0, col0, M, N are the same for all of them).
__device__ __forceinline__ void epilogue_row32(const Epilogue &e, const float (&v)[32], long long row0, int lane, long long col0, int M, int N,
                                               bool vec_ok, int mode, float *tr) {
  if (col0 >= N) return;
  if (vec_ok && col0 + 32 <= N) {
    switch (mode) {
      case 0:
        if (e.stats_kind == 1) epilogue_block32<false, false, false, 1>(e, tr, v, lane, row0, col0, M);
        else epilogue_block32<false, false, false>(e, tr, v, lane, row0, col0, M);
        break;
      case 1:
        if (e.stats_kind == 2) epilogue_block32<false, true, false, 2>(e, tr, v, lane, row0, col0, M);
        else epilogue_block32<false, true, false>(e, tr, v, lane, row0, col0, M);
        break;
      case 2: epilogue_block32<false, false, true>(e, tr, v, lane, row0, col0, M); break;
      default: epilogue_block32<true, true, true>(e, tr, v, lane, row0, col0, M); break;
    }
  } else {
    epilogue_block32_rows(e, tr, v, lane, row0, col0, M, N);
  }
}


}  // namespace myea
