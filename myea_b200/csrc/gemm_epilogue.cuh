// The fused epilogue of the contraction kernels: what happens to the product between the accumulators and global memory
// (bias, skip-connection addend, activation derivative with the normalization folded in, accumulation, column statistics),
// warp-collective over 32-row strips, and element-wise for the kernels that hold single elements.
#pragma once

#include "common.cuh"

namespace myea {

// offset of output row m from e.C: plain pitch, or one of up to four row segments that start at their own offsets
__device__ __forceinline__ long long c_row(const Epilogue &e, long long m) {
  if (e.seg_rows == 0) return m * e.ldc;
  const int s = static_cast<int>(m >= e.seg_rows) + static_cast<int>(m >= 2 * e.seg_rows) + static_cast<int>(m >= 3 * e.seg_rows);
  return (m - s * e.seg_rows) * e.ldc + e.seg_off[s];
}

// The derivative switch has two dozen cases: inlined at every use it makes kernels of many kilobytes that take minutes to
// compile, and a call costs the unrolled epilogues half a kilobyte of spills.  The tensor-core epilogue carries the
// functions below; half_gemm applies the others in a pass of its own.
__host__ __device__ __forceinline__ bool derivative_is_fused(uint32_t af) {
  switch (af) {
    case 0: case MYEA_AF_TANH: case MYEA_AF_SIGMOID: case MYEA_AF_RELU: case MYEA_AF_LEAKY_RELU: case MYEA_AF_ELU: case MYEA_AF_SELU: case MYEA_AF_LINEAR:
    case MYEA_AF_LINEAR_PIECE: case MYEA_AF_LINEAR_PIECE_SYMMETRIC: case MYEA_AF_SOFTMAX: return true;
    default: return false;
  }
}
static __device__ __noinline__ float af_derive_rare(uint32_t af, float z, float y) { return af_derive(af, z, y); }

__device__ __forceinline__ float af_derive_fused(uint32_t af, float z, float y) {   // the functions of derivative_is_fused
  switch (af) {
    case MYEA_AF_TANH: return af_derive(MYEA_AF_TANH, z, y);
    case MYEA_AF_SIGMOID: return af_derive(MYEA_AF_SIGMOID, z, y);
    case MYEA_AF_RELU: return af_derive(MYEA_AF_RELU, z, y);
    case MYEA_AF_LEAKY_RELU: return af_derive(MYEA_AF_LEAKY_RELU, z, y);
    case MYEA_AF_ELU: return af_derive(MYEA_AF_ELU, z, y);
    case MYEA_AF_SELU: return af_derive(MYEA_AF_SELU, z, y);
    default: return 1.0f;
  }
}

template <bool RARE>
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
    v *= RARE ? af_derive_rare(e.deriv_af, pre, y) : af_derive_fused(e.deriv_af, pre, y);
  }
  if (e.accumulate) v += e.C[c_row(e, m) + n];
  return v;
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void add4(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

// The vector path of the epilogue needs 16-byte aligned bases and pitches that are multiples of four floats.
__host__ __device__ __forceinline__ bool epilogue_vector_ok(const Epilogue &e) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(e.C) | reinterpret_cast<uintptr_t>(e.bias) | reinterpret_cast<uintptr_t>(e.addend) |
                         reinterpret_cast<uintptr_t>(e.aux_pre) | reinterpret_cast<uintptr_t>(e.aux_y) |
                         reinterpret_cast<uintptr_t>(e.col_scale) | reinterpret_cast<uintptr_t>(e.col_shift);
  return (bits & 15) == 0 && ((e.ldc | e.ld_addend | e.ld_aux | e.seg_off[0] | e.seg_off[1] | e.seg_off[2] | e.seg_off[3]) & 3) == 0;
}

// Which arrays the derivative of a launch reads decides the variant of the strip epilogue, so that the common ones carry one
// array of loads and two functions.
enum { AUX_NONE = 0, AUX_PRE = 1, AUX_Y = 2, AUX_BOTH = 3 };
template <int AUX>
__device__ __forceinline__ void derive4(uint32_t af, float4 &x, const float4 &z, const float4 &y) {
#define MYEA_DERIVE4(F) x.x *= af_derive(F, z.x, y.x); x.y *= af_derive(F, z.y, y.y); x.z *= af_derive(F, z.z, y.z); x.w *= af_derive(F, z.w, y.w)
  if (AUX == AUX_PRE) {
    if (af == MYEA_AF_RELU) { MYEA_DERIVE4(MYEA_AF_RELU); }
    else { MYEA_DERIVE4(MYEA_AF_LEAKY_RELU); }
  } else if (AUX == AUX_Y) {
    if (af == MYEA_AF_TANH) { MYEA_DERIVE4(MYEA_AF_TANH); }
    else { MYEA_DERIVE4(MYEA_AF_SIGMOID); }
  } else {
    if (af == MYEA_AF_ELU) { MYEA_DERIVE4(MYEA_AF_ELU); }
    else { MYEA_DERIVE4(MYEA_AF_SELU); }
  }
#undef MYEA_DERIVE4
}

// Epilogue of a 32-row x 32-column block, warp-collective: lane l holds row row0 + l (that is how tensor memory hands an
// accumulator to a warp), but global memory wants rows of 128 contiguous bytes.  The block goes through a 32 x 32 float
// staging buffer in shared memory whose 16-byte chunks are swizzled by the row (chunk c of row r lies at c ^ (r & 7): eight
// lanes touch eight different chunks both when a lane writes its row and when it reads a column slot): every lane writes its
// row, then takes one float4 column slot (lane % 8) of the rows lane / 8 + 4 i, so that each global instruction of the warp
// covers four full 128-byte row segments.  The drain warps are two to a scheduler, so what counts is the chain of waits: the
// global reads go out before anything else and the block passes through in one go (in two halves of 16 rows, with a barrier
// more per block, the inference pass of eight 4096-wide layers took 3.33 ms instead of 3.27).
constexpr int TR_WARP_FLOATS = 32 * 32;
__device__ __forceinline__ int tr_at(int r, int chunk) { return r * 32 + ((chunk ^ (r & 7)) << 2); }

template <bool ADD, int AUX, bool ACC, int STATS, typename Stage>
__device__ __forceinline__ void epilogue_block32(const Epilogue &e, float *tr, const Stage &stage, int lane, long long row0, long long col0, int M) {
  const int c4 = (lane & 7) * 4, rsub = lane >> 3;
  const long long n = col0 + c4;
  constexpr bool PRE = (AUX & AUX_PRE) != 0 || STATS == 2, Y = (AUX & AUX_Y) != 0;
  const bool affine = (AUX & AUX_PRE) != 0 && e.col_scale != nullptr;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 bias = e.bias != nullptr ? ld4(e.bias + n) : zero;
  const float4 cs = affine ? ld4(e.col_scale + n) : make_float4(1.f, 1.f, 1.f, 1.f), ch = affine ? ld4(e.col_shift + n) : zero;
  // rows rsub + 4 i of the block; one pointer per array and a step between its rows (in segments every row has a place of its own)
  const int rows = static_cast<int>(min(32ll, static_cast<long long>(M) - row0));
  const long long first = row0 + rsub;
  const bool segments = e.seg_rows != 0;
  float *const c_first = e.C + first * e.ldc + n;
  const long long c_step = 4 * e.ldc;
  auto place = [&](int i) { return segments ? e.C + c_row(e, first + 4 * i) + n : c_first + i * c_step; };
  float4 add[ADD ? 8 : 1], pre[PRE ? 8 : 1], y[Y ? 8 : 1], old[ACC ? 8 : 1];
  const float *const add_first = ADD ? e.addend + first * e.ld_addend + n : nullptr, *const pre_first = PRE ? e.aux_pre + first * e.ld_aux + n : nullptr,
                    *const y_first = Y ? e.aux_y + first * e.ld_aux + n : nullptr;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const bool in = rsub + 4 * i < rows;
    if (ADD) add[i] = in ? ld4(add_first + i * (4 * e.ld_addend)) : zero;
    if (PRE) pre[i] = in ? ld4(pre_first + i * (4 * e.ld_aux)) : zero;
    if (Y) y[i] = in ? ld4(y_first + i * (4 * e.ld_aux)) : zero;
    if (ACC) old[i] = in ? ld4(place(i)) : zero;
  }
  // column statistics of this 32 x 32 block: this lane's four columns over its eight rows first
  float4 st0 = zero, st1 = zero;
  const float4 mu = (STATS == 2 && e.col_mean != nullptr) ? ld4(e.col_mean + n) : zero;
  __syncwarp();   // the block before has been read
  stage(tr);
  __syncwarp();
  constexpr bool AHEAD = ADD + PRE + Y + ACC <= 1;   // (the rows wait in registers where there is room beside the other arrays)
  float4 v[AHEAD ? 8 : 1];
  if constexpr (AHEAD) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const float4 *>(tr + tr_at(rsub + 4 * i, lane & 7));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4 x = AHEAD ? v[i] : *reinterpret_cast<const float4 *>(tr + tr_at(rsub + 4 * i, lane & 7));
    add4(x, bias);
    if (ADD) add4(x, add[i]);
    if (AUX != AUX_NONE) {
      float4 z = zero;
      if (PRE) {
        const float4 p = pre[i];
        z = make_float4(p.x * cs.x + ch.x, p.y * cs.y + ch.y, p.z * cs.z + ch.z, p.w * cs.w + ch.w);
      }
      derive4<AUX>(e.deriv_af, x, z, Y ? y[i] : zero);
    }
    if (ACC) add4(x, old[i]);
    if (rsub + 4 * i < rows) {
      *reinterpret_cast<float4 *>(place(i)) = x;
      if (STATS == 1) {
        add4(st0, x);
        st1.x = fmaf(x.x, x.x, st1.x); st1.y = fmaf(x.y, x.y, st1.y); st1.z = fmaf(x.z, x.z, st1.z); st1.w = fmaf(x.w, x.w, st1.w);
      }
      if (STATS == 2) {
        const float4 p = pre[i];  // the raw array the derivative was taken on (before the folded normalization)
        add4(st0, x);
        st1.x = fmaf(x.x, p.x - mu.x, st1.x); st1.y = fmaf(x.y, p.y - mu.y, st1.y); st1.z = fmaf(x.z, p.z - mu.z, st1.z); st1.w = fmaf(x.w, p.w - mu.w, st1.w);
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
// derivatives of LSTM layers land inside the reference's per-block parameter layout, whose row pitch is odd), for the
// ragged right edge and for combinations without a variant of their own: staged through the same buffer, then lane l takes
// column col0 + l of one row after the other, so a warp's accesses still cover one contiguous row segment each.
template <typename Stage>
__device__ __forceinline__ void epilogue_block32_rows(const Epilogue &e, float *tr, const Stage &stage, int lane, long long row0, long long col0, int M, int N) {
  const long long n = col0 + lane;
  const bool plain = e.bias == nullptr && e.addend == nullptr && e.deriv_af == 0u;
  __syncwarp();
  stage(tr);
  __syncwarp();
  auto at = [&](int r) { return tr[tr_at(r, lane >> 2) + (lane & 3)]; };
  if (plain && e.accumulate) {
    // C += product and nothing else (weight derivatives): 16 old row segments are requested together - one after the other,
    // their latency (rows of an LSTM layer's weight derivatives lie a whole block apart) is what the epilogue of a tile takes
#pragma unroll 1
    for (int h = 0; h < 32; h += 16) {
      float old[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const long long m = row0 + h + r;
        old[r] = (m < M && n < N) ? e.C[c_row(e, m) + n] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const long long m = row0 + h + r;
        if (m < M && n < N) e.C[c_row(e, m) + n] = at(h + r) + old[r];
      }
    }
  } else if (plain) {
#pragma unroll 16
    for (int r = 0; r < 32; ++r) {
      const long long m = row0 + r;
      if (m < M && n < N) e.C[c_row(e, m) + n] = at(r);
    }
  } else {
#pragma unroll 1
    for (int r = 0; r < 32; ++r) {
      const long long m = row0 + r;
      if (m < M && n < N) e.C[c_row(e, m) + n] = epilogue_value<false>(e, at(r), m, n);
    }
  }
}

// Variant of the strip epilogue for a launch; chosen on the host.
enum { EPI_PLAIN = 0, EPI_PLAIN_STATS, EPI_ACC, EPI_ADD, EPI_PRE, EPI_PRE_STATS, EPI_Y, EPI_Y_STATS, EPI_BOTH, EPI_BOTH_STATS, EPI_ADD_PRE, EPI_ADD_Y, EPI_ADD_BOTH, EPI_ROWS };
inline int epilogue_variant(const Epilogue &e) {
  if (!epilogue_vector_ok(e)) return EPI_ROWS;
  const bool derives = e.deriv_af != 0u && (e.aux_pre != nullptr || e.aux_y != nullptr) &&
                       (af_derive_reads_summation(e.deriv_af) || af_derive_reads_value(e.deriv_af));
  if (e.accumulate) return e.addend == nullptr && !derives && e.stats_kind == 0 ? EPI_ACC : EPI_ROWS;
  if (!derives) {
    if (e.addend != nullptr) return e.stats_kind == 0 ? EPI_ADD : EPI_ROWS;
    return e.stats_kind == 1 ? EPI_PLAIN_STATS : (e.stats_kind == 2 ? EPI_ROWS : EPI_PLAIN);
  }
  const bool pre = af_derive_reads_summation(e.deriv_af), y = af_derive_reads_value(e.deriv_af);
  const int which = pre && y ? 2 : (y ? 1 : 0);
  if (e.addend != nullptr) return e.stats_kind == 0 ? EPI_ADD_PRE + which : EPI_ROWS;
  return EPI_PRE + 2 * which + (e.stats_kind == 2 ? 1 : 0);
}

// 32 rows x NCOLS columns held as one row per lane; warp-collective.  The 32-column blocks go one after the other through
// one copy of the code: the block's registers are picked by a uniform switch in front of the staging stores.
template <int NCOLS>
__device__ __forceinline__ void epilogue_strip(const Epilogue &e, int variant, float *tr, const float (&sum)[NCOLS], int lane, long long row0, long long col_base, int M, int N) {
  __builtin_assume(__isShared(tr));   // (its address went through an integer on the way here)
#pragma unroll 1
  for (int jc = 0; jc < NCOLS / 32; ++jc) {
    const long long col0 = col_base + jc * 32;
    if (col0 >= N) break;
    auto stage = [&](float *t) {
#define MYEA_STAGE(J)                                                                                                        \
  if (J * 32 < NCOLS && jc == J) {                                                                                           \
    _Pragma("unroll") for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(t + tr_at(lane, j)) =                                 \
        make_float4(sum[(J * 32 + 4 * j) % NCOLS], sum[(J * 32 + 4 * j + 1) % NCOLS], sum[(J * 32 + 4 * j + 2) % NCOLS], sum[(J * 32 + 4 * j + 3) % NCOLS]); \
  }
      MYEA_STAGE(0) MYEA_STAGE(1) MYEA_STAGE(2) MYEA_STAGE(3)
#undef MYEA_STAGE
    };
    const int v = col0 + 32 <= N ? variant : EPI_ROWS;
    switch (v) {
      case EPI_PLAIN: epilogue_block32<false, AUX_NONE, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_PLAIN_STATS: epilogue_block32<false, AUX_NONE, false, 1>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_ACC: epilogue_block32<false, AUX_NONE, true, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_ADD: epilogue_block32<true, AUX_NONE, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_PRE: epilogue_block32<false, AUX_PRE, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_PRE_STATS: epilogue_block32<false, AUX_PRE, false, 2>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_Y: epilogue_block32<false, AUX_Y, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_Y_STATS: epilogue_block32<false, AUX_Y, false, 2>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_BOTH: epilogue_block32<false, AUX_BOTH, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_BOTH_STATS: epilogue_block32<false, AUX_BOTH, false, 2>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_ADD_PRE: epilogue_block32<true, AUX_PRE, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_ADD_Y: epilogue_block32<true, AUX_Y, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      case EPI_ADD_BOTH: epilogue_block32<true, AUX_BOTH, false, 0>(e, tr, stage, lane, row0, col0, M); break;
      default: epilogue_block32_rows(e, tr, stage, lane, row0, col0, M, N); break;
    }
  }
}

}  // namespace myea
