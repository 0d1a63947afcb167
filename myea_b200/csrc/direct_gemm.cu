// Contractions of small and middle sizes straight from fp32 operands:  C[M,N] (+)= A[M,K] * B[N,K]^T, several per launch.
//
// The kernels of half_gemm.cu read operand panels that split passes have written before: three launches and two extra trips
// through L2 per product, which is nothing beside a large product and everything beside a small one (a training step of
// a 64-256-256-10 network on 128 rows spent 236 us in 37 launches around 0.06 GFLOP, and its tiles of 128 x 128 kept four
// SMs busy).  Here the operands are read as they lie (rows or columns contiguous, any pitch), split in registers and
// stored as the tensor core wants them, and the result leaves through the same fused epilogue, plus the layer's
// activation and dropout; the weight derivatives of a whole network are one launch.
//
//   tile      128 x 64 per CTA of 8 warps, two CTAs per SM, 32 of K per stage, 2 stages of 48 KB.  At these sizes a
//             product is bounded by latency, so tiles are small and the K range of a tile is cut over the CTAs of a cluster
//             (1, 2, 4 or 8) until the grid fills the chip; partial tiles meet in distributed shared memory and are added
//             in rank order (bitwise repeatable)
//   stage     every thread splits 24 elements: 8 consecutive K of three rows, fetched into registers while the stage before
//             is converted.  hi (TF32) and the cross-term group (bf16, see split_group) go into K-major tiles with the
//             128-byte swizzle; one thread then issues the eight tcgen05.mma of the stage.  (Warp-level mma.sync was
//             built first: 512^3 took 12 us instead of 17 with panels; its TF32 rate on this chip is below what the
//             precision needs - three TF32 products run no faster than plain FMAs.)
//   sums      three rotating accumulators for hi*hi and one for the cross terms
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "half_panels.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <mutex>

namespace myea {

constexpr int DG_M = 128, DG_N = 64, DG_THREADS = 256;
constexpr int DG_A_BYTES = DG_M * BK * 4, DG_B_BYTES = DG_N * BK * 4;       // one panel (hi or cross) of a stage
constexpr int DG_STAGE_BYTES = 2 * DG_A_BYTES + 2 * DG_B_BYTES;             // A hi, A cross, B hi, B cross
constexpr int DG_STAGES = 2, DG_MAIN = 3, DG_TMEM_COLS = 256;
static_assert((DG_MAIN + 1) * DG_N <= DG_TMEM_COLS, "accumulators exceed the allocation");
constexpr int DG_RED_PITCH = DG_N + 4;      // partial tile [128][68], then row sums [2][128]: over the stages, which are free by then
static_assert((DG_M * DG_RED_PITCH + 2 * DG_M) * 4 <= DG_STAGES * DG_STAGE_BYTES, "the partial tile lies over the stages");
constexpr int DG_BAR_OFFSET = DG_STAGES * DG_STAGE_BYTES;
constexpr int DG_SMEM = DG_BAR_OFFSET + 64 + 1024;
constexpr int DG_MAX_ITEMS = 12;
constexpr int FG_M = 32, FG_N = 32;          // tile of the kernel that multiplies with plain FMAs
constexpr int FG_K = 256;                    // K it holds in shared memory at a time

// x rounded to TF32, half away from zero, on the integer pipe: cvt.rna.tf32 gives the same bits at a quarter of the rate
// (it and single bf16 conversions kept the pipe of special functions busy: 14 instructions per split element, now 4).
// A NaN leaves its trace in the low part x - round_tf32(x).
__device__ __forceinline__ float round_tf32(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
// two values as a bf16 pair, a in the lower half
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

struct DirectProblem {
  const float *a, *b;
  long long lda, ldb;    // pitch of the non-contiguous index
  int M, N, K;
  int tiles_n, first_tile;
  int a_vec, b_vec;      // 16-byte copies possible
  int c_vec;             // 16-byte accesses possible in the epilogue
  float *row_sum;
  Epilogue epi;
};
template <int MAX> struct DirectGroup {   // kernel argument: 400 bytes for a single product, 5 KB for a group
  int count;
  DirectProblem p[MAX];
};

// One thread's 8 consecutive K elements of one operand row, stage after stage.  T: the rows are contiguous in memory (pitch
// ld between K steps), a warp's lanes take consecutive rows; else K is contiguous.  Rows past the matrix repeat its last
// row (what they produce is never stored); K elements past its end are zeros.  WIDE: whole sectors at once where they are aligned.
template <bool T, bool WIDE>
struct DgReader {
  const float *p;     // element (row, k)
  long long ld, advance;
  int k, K;
  bool vec;
  uint32_t at;        // where the group lies in a panel of a stage: rows of 128 bytes, 16-byte chunks swizzled by the row
  __device__ __forceinline__ DgReader(const float *src, long long pitch, int tile_row, int row0, int rows, int group, int k0, int K_, bool vec16)
      : ld(pitch), advance(T ? BK * pitch : BK), k(k0 + 8 * group), K(K_), vec(vec16) {
    const int row = min(row0 + tile_row, rows - 1);
    p = src + (T ? static_cast<long long>(k) * pitch + row : static_cast<long long>(row) * pitch + k);
    at = static_cast<uint32_t>(tile_row * 128 + (((2 * group) ^ (tile_row & 7)) * 16));
  }
  __device__ __forceinline__ void fetch(float (&v)[8]) {
    if (k + 8 <= K) {
      if (T) {
        const float *q = p;
#pragma unroll
        for (int j = 0; j < 8; ++j, q += ld) v[j] = *q;
      } else if (vec) {
        if (WIDE) {
          ld8(v, p, 8, true);
        } else {
          const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
          v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = p[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = k + j < K ? p[T ? j * ld : j] : 0.f;
    }
    p += advance;
    k += BK;
  }
};

// One group of 8 K elements as 8 TF32 values and the 8 words of a cross-term group: 16 bf16, [lo x8 | hi x8] for operand A
// (ROLE 0) and [hi x8 | lo x8] for operand B (ROLE 1), so that one bf16 instruction (K = 16) of an A group with a B group gives
// lo_a*hi_b + hi_a*lo_b
template <int ROLE>
__device__ __forceinline__ void split_group(const float (&v)[8], float (&hi)[8], uint32_t (&cross)[8]) {
  float lo[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    hi[j] = round_tf32(v[j]);
    lo[j] = v[j] - hi[j];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t l = pack_bf16(lo[2 * j], lo[2 * j + 1]), h = pack_bf16(hi[2 * j], hi[2 * j + 1]);
    cross[j] = ROLE ? h : l;
    cross[4 + j] = ROLE ? l : h;
  }
}
// 8 elements as a hi and a cross group into a stage
template <int ROLE>
__device__ __forceinline__ void dg_store8(uint8_t *hi, uint8_t *cross, uint32_t at, const float (&v)[8]) {
  float h[8];
  uint32_t x[8];
  split_group<ROLE>(v, h, x);
  *reinterpret_cast<float4 *>(hi + at) = make_float4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4 *>(hi + (at ^ 16u)) = make_float4(h[4], h[5], h[6], h[7]);
  *reinterpret_cast<uint4 *>(cross + at) = make_uint4(x[0], x[1], x[2], x[3]);
  *reinterpret_cast<uint4 *>(cross + (at ^ 16u)) = make_uint4(x[4], x[5], x[6], x[7]);
}

// Steps of the epilogue on VEC adjacent columns of NB rows, for dg_finish and sg_finish
template <int VEC>
__device__ __forceinline__ void ld_cols(float (&d)[VEC], const float *src) {
  if constexpr (VEC == 4) { const float4 t = *reinterpret_cast<const float4 *>(src); d[0] = t.x; d[1] = t.y; d[2] = t.z; d[3] = t.w; }
  else d[0] = *src;
}
template <int VEC>
__device__ __forceinline__ void st_cols(float *dst, const float (&d)[VEC]) {
  if constexpr (VEC == 4) *reinterpret_cast<float4 *>(dst) = make_float4(d[0], d[1], d[2], d[3]);
  else *dst = d[0];
}
// what dropout leaves of the columns from n on
template <int VEC>
__device__ __forceinline__ void dg_factors(const Epilogue &e, int n, float (&factor)[VEC]) {
#pragma unroll
  for (int k = 0; k < VEC; ++k) factor[k] = (e.act_mask != nullptr && e.act_mask[n + k] == 0) ? 0.f : e.act_scale;
}
// take(row, column, slope): the activation's derivative at each element
template <int NB, int VEC, typename Take>
__device__ __forceinline__ void dg_derive(const Epilogue &e, const float (&pre)[NB][VEC], const float (&y)[NB][VEC], const float (&cs)[VEC], const float (&ch)[VEC], Take take) {
  auto derive = [&](auto f) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int k = 0; k < VEC; ++k) take(b, k, f(e.aux_pre != nullptr ? pre[b][k] * cs[k] + ch[k] : 0.f, e.aux_y != nullptr ? y[b][k] : 0.f));
  };
  switch (e.deriv_af) {
    case MYEA_AF_TANH: derive([](float z, float w) { return af_derive(MYEA_AF_TANH, z, w); }); break;
    case MYEA_AF_RELU: derive([](float z, float w) { return af_derive(MYEA_AF_RELU, z, w); }); break;
    default: { const uint32_t af = e.deriv_af; derive([af](float z, float w) { return af_derive_rare(af, z, w); }); break; }
  }
}
// activation and dropout in place
template <int NB, int VEC>
__device__ __forceinline__ void dg_fire(const Epilogue &e, float (&v)[NB][VEC], const float (&factor)[VEC]) {
  auto fire = [&](auto f) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int k = 0; k < VEC; ++k) { const float t = f(v[b][k]); v[b][k] = factor[k] != 0.f ? t * factor[k] : 0.f; }
  };
  switch (e.act_af) {
    case MYEA_AF_TANH: fire([](float z) { return af_fire(MYEA_AF_TANH, z); }); break;
    case MYEA_AF_RELU: fire([](float z) { return af_fire(MYEA_AF_RELU, z); }); break;
    case MYEA_AF_LINEAR: fire([](float z) { return z; }); break;
    default: { const uint32_t af = e.act_af; fire([af](float z) { return af_fire_rare(af, z); }); break; }
  }
}

// What this CTA finishes of its tile: rows [first, first + count), summed over the CTAs of the cluster in rank order, through
// the epilogue.  A thread keeps VEC adjacent columns and takes NB rows at a time, all their loads before the first use: with
// a row at a time this part was latency after latency and took longer than the products (29 of 31 us at K = 10).
// TN: columns of the tile; PARTS: partial tiles of FG_M rows in this CTA's own shared memory, one behind the other (S == 1).
template <int TN, int PARTS, int VEC, int NB>
__device__ __forceinline__ void dg_finish(const DirectProblem &p, const float *partial, uint32_t S, int first, int count, int m0, int n0) {
  constexpr int LANES = TN / VEC, STEP = DG_THREADS / LANES, PITCH = TN + 4;
  using Vec = float[VEC];
  const Epilogue &e = p.epi;
  const int c = (static_cast<int>(threadIdx.x) % LANES) * VEC, n = n0 + c;
  if (n >= p.N) return;
  const bool affine = e.deriv_af != 0u && e.aux_pre != nullptr && e.col_scale != nullptr;
  Vec bias = {}, cs, ch = {};
#pragma unroll
  for (int k = 0; k < VEC; ++k) cs[k] = 1.f;
  if (e.bias != nullptr) ld_cols(bias, e.bias + n);
  if (affine) { ld_cols(cs, e.col_scale + n); ld_cols(ch, e.col_shift + n); }
  float factor[VEC];
  if (e.act_out != nullptr) dg_factors<VEC>(e, n, factor);
  const int end = min(first + count, p.M - m0);
#pragma unroll 1
  for (int r0 = first + static_cast<int>(threadIdx.x) / LANES; r0 < end; r0 += NB * STEP) {
    Vec v[NB], add[NB], pre[NB], y[NB], old[NB];
    float *dst[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int r = min(r0 + b * STEP, end - 1);   // rows past the end repeat the last one and are not stored
      const long long m = m0 + r;
      dst[b] = e.C + c_row(e, m) + n;
#pragma unroll
      for (int k = 0; k < VEC; ++k) v[b][k] = 0.f;
      if (e.addend != nullptr) ld_cols(add[b], e.addend + m * e.ld_addend + n);
      if (e.deriv_af != 0u && e.aux_pre != nullptr) ld_cols(pre[b], e.aux_pre + m * e.ld_aux + n);
      if (e.deriv_af != 0u && e.aux_y != nullptr) ld_cols(y[b], e.aux_y + m * e.ld_aux + n);
      if (e.accumulate) ld_cols(old[b], dst[b]);
      if (S == 1) {
#pragma unroll
        for (int q = 0; q < PARTS; ++q) {
          Vec t;
          ld_cols(t, partial + (q * FG_M + r) * PITCH + c);   // (one part: row r of it)
#pragma unroll
          for (int k = 0; k < VEC; ++k) v[b][k] += t[k];
        }
      }
    }
    if (PARTS == 1 && S > 1) {
#pragma unroll 2
      for (uint32_t q = 0; q < S; ++q) {
        const uint32_t base = ptx::map_to_cta(ptx::smem_u32(partial), q);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const uint32_t at = base + (min(r0 + b * STEP, end - 1) * PITCH + c) * 4;
          if constexpr (VEC == 4) {
            const float4 t = ptx::ld_cluster_f4(at);
            v[b][0] += t.x; v[b][1] += t.y; v[b][2] += t.z; v[b][3] += t.w;
          } else {
            float t;
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t) : "r"(at) : "memory");
            v[b][0] += t;
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        v[b][k] += bias[k];
        if (e.addend != nullptr) v[b][k] += add[b][k];
      }
    }
    if (e.deriv_af != 0u) dg_derive<NB, VEC>(e, pre, y, cs, ch, [&](int b, int k, float slope) { v[b][k] *= slope; });
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (r0 + b * STEP >= end) break;
      if (e.accumulate) {
#pragma unroll
        for (int k = 0; k < VEC; ++k) v[b][k] += old[b][k];
      }
      st_cols(dst[b], v[b]);
    }
    if (e.act_out != nullptr) {
      dg_fire<NB, VEC>(e, v, factor);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (r0 + b * STEP >= end) break;
        st_cols(e.act_out + (dst[b] - e.C), v[b]);
      }
    }
  }
}

template <bool AT, bool BT, int MAX, bool WIDE>
__global__ void __launch_bounds__(DG_THREADS, 2) direct_gemm_kernel(const __grid_constant__ DirectGroup<MAX> g, int *error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t *free_bar = reinterpret_cast<uint64_t *>(smem + DG_BAR_OFFSET);  // [2] the products of a stage have been computed
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(free_bar + DG_STAGES);
  uint32_t S;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
  const uint32_t rank = ptx::cluster_ctarank();
  const int tile = static_cast<int>(blockIdx.x / S);
  int pi = 0;
#pragma unroll 1
  while (pi + 1 < g.count && tile >= g.p[pi + 1].first_tile) ++pi;
  const DirectProblem &p = g.p[pi];
  const int tl = tile - p.first_tile;
  const int tm = tl / p.tiles_n, tn = tl - tm * p.tiles_n;
  const int m0 = tm * DG_M, n0 = tn * DG_N;
  const int steps = (p.K + BK - 1) / BK;
  const int per = (steps + static_cast<int>(S) - 1) / static_cast<int>(S);
  const int s0 = min(static_cast<int>(rank) * per, steps), n_steps = min(s0 + per, steps) - s0;
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const bool want_sum = AT && p.row_sum != nullptr && tn == 0;
  if (tid == 0) {
    for (int s = 0; s < DG_STAGES; ++s) ptx::mbar_init(&free_bar[s], 1);
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_holder, DG_TMEM_COLS);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  grid_dependency_wait();
  grid_dependency_release();

  // this thread's share of a stage: rows (a0, group ag0), (a1, ag1) of A and (b0, bg) of B
  const int a0 = AT ? (tid & 127) : (tid >> 2), ag0 = AT ? (tid >> 7) : (tid & 3);
  const int a1 = AT ? a0 : a0 + 64, ag1 = AT ? ag0 + 2 : ag0;
  const int b0 = BT ? (tid & 63) : (tid >> 2), bg = BT ? (tid >> 6) : (tid & 3);
  // two register sets: the loads of stage i + 2 leave when stage i has been stored, so that their way to L2 and back
  // runs beside the conversion of stage i + 1
  float va0[2][8], va1[2][8], vb[2][8];
  DgReader<AT, WIDE> ra0(p.a, p.lda, a0, m0, p.M, ag0, s0 * BK, p.K, p.a_vec != 0), ra1(p.a, p.lda, a1, m0, p.M, ag1, s0 * BK, p.K, p.a_vec != 0);
  DgReader<BT, WIDE> rb(p.b, p.ldb, b0, n0, p.N, bg, s0 * BK, p.K, p.b_vec != 0);
  auto fetch = [&](float (&x0)[8], float (&x1)[8], float (&xb)[8]) { ra0.fetch(x0); ra1.fetch(x1); rb.fetch(xb); };
  float rs = 0.f;   // thread: row tid & 127, half of the K groups of every stage
  bool ok = true;
  if (n_steps > 0) fetch(va0[0], va1[0], vb[0]);
  if (n_steps > 1) fetch(va0[1], va1[1], vb[1]);
#pragma unroll 1
  for (int i2 = 0; i2 < n_steps; i2 += 2) {
#pragma unroll
    for (int s = 0; s < DG_STAGES; ++s) {
      const int i = i2 + s;
      if (i >= n_steps) break;
      uint8_t *st = smem + s * DG_STAGE_BYTES;
      if (i >= DG_STAGES && !ptx::mbar_wait(&free_bar[s], static_cast<uint32_t>((i >> 1) - 1) & 1u)) ok = false;
      dg_store8<0>(st, st + DG_A_BYTES, ra0.at, va0[s]);
      dg_store8<0>(st, st + DG_A_BYTES, ra1.at, va1[s]);
      dg_store8<1>(st + 2 * DG_A_BYTES, st + 2 * DG_A_BYTES + DG_B_BYTES, rb.at, vb[s]);
      if (want_sum) {
#pragma unroll
        for (int j = 0; j < 8; ++j) rs += va0[s][j] + va1[s][j];
      }
      if (i + 2 < n_steps) fetch(va0[s], va1[s], vb[s]);
      ptx::fence_proxy_async();
      __syncthreads();
      if (tid == 0 && ok) {
        ptx::tc_fence_after();
        const uint32_t base = ptx::smem_u32(st);
        const uint64_t a_hi = make_smem_desc(base), a_x = make_smem_desc(base + DG_A_BYTES);
        const uint64_t b_hi = make_smem_desc(base + 2 * DG_A_BYTES), b_x = make_smem_desc(base + 2 * DG_A_BYTES + DG_B_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t koff = static_cast<uint64_t>((k * UMMA_K * 4) >> 4);
          const int step = i * (BK / UMMA_K) + k;
          ptx::mma_bf16(tmem + DG_MAIN * DG_N, a_x + koff, b_x + koff, make_idesc_bf16(DG_M, DG_N), step > 0 ? 1u : 0u);
          ptx::mma_tf32(tmem + static_cast<uint32_t>((step % DG_MAIN) * DG_N), a_hi + koff, b_hi + koff, make_idesc_tf32(DG_M, DG_N), step >= DG_MAIN ? 1u : 0u);
        }
        ptx::tc_commit(&free_bar[s]);
      }
    }
  }
  // the last commit covers everything issued before it
  float *partial = reinterpret_cast<float *>(smem);
  if (n_steps > 0 && !ptx::mbar_wait(&free_bar[(n_steps - 1) & 1], static_cast<uint32_t>((n_steps - 1) >> 1) & 1u)) ok = false;
  if (!ok && lane == 0) atomicCAS(error_flag, 0, 111);
  ptx::tc_fence_after();
  {
    // accumulators -> partial tile: warp = 32 rows (warp % 4) x 32 columns (warp / 4)
    const int q = warp & 3, half = warp >> 2;
    float sum[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) sum[j] = 0.f;
    const int filled = min(DG_MAIN, n_steps * (BK / UMMA_K));   // 0 or all of them: a stage has four K steps
#pragma unroll
    for (int acc = 0; acc <= DG_MAIN; ++acc) {
      if (filled == 0) break;
      uint32_t r[32];
      ptx::tmem_ld_32x32(tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>((DG_MAIN - acc) * DG_N + half * 32), r);  // cross terms first
      ptx::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[j] += __uint_as_float(r[j]);
    }
    float *d = partial + (q * 32 + lane) * DG_RED_PITCH + half * 32;
#pragma unroll
    for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(d + 4 * j) = make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
  }
  if (want_sum) partial[DG_M * DG_RED_PITCH + tid] = rs;   // [2][128]
  ptx::tc_fence_before();
  if (S > 1) ptx::cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, DG_TMEM_COLS);
  }
  const int my_rows = DG_M / static_cast<int>(S), first = static_cast<int>(rank) * my_rows;
  if (p.c_vec) dg_finish<DG_N, 1, 4, 2>(p, partial, S, first, my_rows, m0, n0);
  else dg_finish<DG_N, 1, 1, 8>(p, partial, S, first, my_rows, m0, n0);
  if (want_sum) {
    for (int r = first + tid; r < first + my_rows; r += DG_THREADS) {
      if (m0 + r >= p.M) continue;
      const uint32_t at = ptx::smem_u32(partial + DG_M * DG_RED_PITCH + r);
      float v = 0.f;
      for (uint32_t q = 0; q < S; ++q) {
        float x[2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[k]) : "r"(ptx::map_to_cta(at + k * DG_M * 4, q)) : "memory");
        v += x[0] + x[1];
      }
      p.row_sum[m0 + r] += v;
    }
  }
  if (S > 1) ptx::cluster_sync_all();  // a peer may still be reading this CTA's partial tile
}

// ---------------------------------------------------------------------------------------------------------
// The smallest products with plain FMAs.  A tensor-core tile pays for tensor memory, barriers, conversion, a cluster and its
// exchange before anything else: 128 x 256 x 256 takes it 6.8 us (here 5.2), of which the products are a tenth.  Here a CTA owns
// 32 x 32 outputs, fetches both operands' rows for up to 256 of K at once (16 loads of 16 bytes per thread in flight: one trip
// to L2), and its 8 warps walk interleaved groups of four K each with 4 x 8 sums per lane; the 8 partial tiles are added in warp
// order in shared memory (bitwise repeatable).  Bound by latency, then by shared-memory reads and FMA issue (11 ns per K): a long K of
// few tiles is cut over the CTAs of a cluster, whose tiles are added in rank order through distributed shared memory.
// Operand rows contiguous in K lie as [row][FG_K + 4] (lanes read rows rg + 8 i: eight different 16-byte chunks), operands
// read through their columns as [k][32].
// ---------------------------------------------------------------------------------------------------------
constexpr int FG_PITCH = FG_K + 4;
constexpr int FG_OP_FLOATS = 32 * FG_PITCH;               // one operand
constexpr int FG_TILE_FLOATS = FG_M * (FG_N + 4);
constexpr int FG_RED_FLOATS = 9 * FG_TILE_FLOATS + 9 * FG_M;   // the warps' partial tiles and their sum, the warps' row sums and theirs; over the operands
constexpr int FG_SMEM = (2 * FG_OP_FLOATS > FG_RED_FLOATS ? 2 * FG_OP_FLOATS : FG_RED_FLOATS) * 4;

// rows row0 .. row0 + 31 (past `rows`: the last one again), K elements k0 .. k0 + kc - 1 (zeros up to a multiple of 4)
template <bool T>
__device__ __forceinline__ void fg_fetch(float *s, const float *src, long long ld, int row0, int rows, int k0, int kc, bool vec) {
  const int tid = static_cast<int>(threadIdx.x), kz = (kc + 3) & ~3;
  if (T) {
    // [k][32]: lanes take consecutive rows
    if (vec && row0 + 32 <= rows) {
      const int c = (tid & 7) * 4, kk0 = tid >> 3;   // 32 K rows per round
      float4 v[8];
#pragma unroll
      for (int i = 0; i < FG_K / 32; ++i) {
        const int kk = kk0 + 32 * i;
        if (kk < kc) v[i] = *reinterpret_cast<const float4 *>(src + static_cast<long long>(k0 + kk) * ld + row0 + c);
        else v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < FG_K / 32; ++i) {
        const int kk = kk0 + 32 * i;
        if (kk < kz) *reinterpret_cast<float4 *>(s + kk * 32 + c) = v[i];
      }
    } else {
      const int r = tid & 31, row = min(row0 + r, rows - 1);
      const float *q = src + static_cast<long long>(k0) * ld + row;
      for (int base = 0; base < kz; base += 64) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int kk = base + (tid >> 5) + 8 * i;
          v[i] = kk < kc ? q[static_cast<long long>(kk) * ld] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int kk = base + (tid >> 5) + 8 * i;
          if (kk < kz) s[kk * 32 + r] = v[i];
        }
      }
    }
  } else if (vec && (kc & 3) == 0) {
    // [row][FG_PITCH]: lanes take consecutive 16-byte chunks of a row (a whole row of 256 by two warps)
    const int c = (tid & 63) * 4, r0 = tid >> 6;
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = min(row0 + r0 + 4 * i, rows - 1);
      if (c < kc) v[i] = *reinterpret_cast<const float4 *>(src + static_cast<long long>(row) * ld + k0 + c);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c < kc) *reinterpret_cast<float4 *>(s + (r0 + 4 * i) * FG_PITCH + c) = v[i];
  } else {
    const int lane = tid & 31, r0 = tid >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = min(row0 + r0 + 8 * i, rows - 1);
      const float *q = src + static_cast<long long>(row) * ld + k0;
      float v[FG_K / 32];
#pragma unroll
      for (int j = 0; j < FG_K / 32; ++j) v[j] = lane + 32 * j < kc ? q[lane + 32 * j] : 0.f;
#pragma unroll
      for (int j = 0; j < FG_K / 32; ++j)
        if (lane + 32 * j < kz) s[(r0 + 8 * i) * FG_PITCH + lane + 32 * j] = v[j];
    }
  }
}

// CUT: the CTAs of a cluster share a tile
template <bool AT, bool BT, int MAX, bool CUT>
__global__ void __launch_bounds__(DG_THREADS, 2) fma_gemm_kernel(const __grid_constant__ DirectGroup<MAX> g) {
  extern __shared__ float fg_smem[];
  float *sa = fg_smem, *sb = fg_smem + FG_OP_FLOATS;
  uint32_t S = 1, rank = 0;
  if constexpr (CUT) {
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
    rank = ptx::cluster_ctarank();
  }
  const int tile = static_cast<int>(CUT ? blockIdx.x / S : blockIdx.x);
  int pi = 0;
#pragma unroll 1
  while (pi + 1 < g.count && tile >= g.p[pi + 1].first_tile) ++pi;
  const DirectProblem &p = g.p[pi];
  const int tl = tile - p.first_tile;
  const int tm = tl / p.tiles_n, tn = tl - tm * p.tiles_n;
  const int m0 = tm * FG_M, n0 = tn * FG_N;
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int rg = lane >> 2, cg = lane & 3;   // rows rg + 8 i or 4 rg + i, columns cg + 4 j or 8 cg + j
  const bool want_sum = AT && p.row_sum != nullptr && tn == 0;
  float acc[4][8] = {};
  float rs = 0.f;
  grid_dependency_wait();
  grid_dependency_release();
  int k_begin = 0, k_end = p.K;
  if constexpr (CUT) {
    const int share = ((p.K + static_cast<int>(S) - 1) / static_cast<int>(S) + 3) & ~3;
    k_begin = min(static_cast<int>(rank) * share, p.K);
    k_end = min(k_begin + share, p.K);
  }
#pragma unroll 1
  for (int k0 = k_begin; k0 < k_end; k0 += FG_K) {
    const int kc = min(FG_K, k_end - k0);
    if (k0 > k_begin) __syncthreads();
    fg_fetch<AT>(sa, p.a, p.lda, m0, p.M, k0, kc, p.a_vec != 0);
    fg_fetch<BT>(sb, p.b, p.ldb, n0, p.N, k0, kc, p.b_vec != 0);
    __syncthreads();
    if (want_sum)
      for (int k = warp; k < kc; k += 8) rs += sa[k * 32 + lane];
#pragma unroll 2
    for (int k = warp * 4; k < kc; k += 32) {
      float a[4][4], b[4][8];   // [row][k], [k][column]
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 t = *reinterpret_cast<const float4 *>(AT ? sa + (k + i) * 32 + rg * 4 : sa + (rg + 8 * i) * FG_PITCH + k);
        if (AT) { a[0][i] = t.x; a[1][i] = t.y; a[2][i] = t.z; a[3][i] = t.w; }
        else { a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w; }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (BT) {
          const float4 t = *reinterpret_cast<const float4 *>(sb + (k + (i >> 1)) * 32 + cg * 8 + (i & 1) * 4);
          b[i >> 1][(i & 1) * 4] = t.x; b[i >> 1][(i & 1) * 4 + 1] = t.y; b[i >> 1][(i & 1) * 4 + 2] = t.z; b[i >> 1][(i & 1) * 4 + 3] = t.w;
        } else {
          const float4 t = *reinterpret_cast<const float4 *>(sb + (cg + 4 * i) * FG_PITCH + k);
          b[0][i] = t.x; b[1][i] = t.y; b[2][i] = t.z; b[3][i] = t.w;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i][kk], b[kk][j], acc[i][j]);
    }
  }
  __syncthreads();   // the operands have been read: the partial tiles take their place
  float *part = fg_smem + warp * FG_TILE_FLOATS;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float *d = part + (AT ? rg * 4 + i : rg + 8 * i) * (FG_N + 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[BT ? cg * 8 + j : cg + 4 * j] = acc[i][j];
  }
  float *sums = fg_smem + 9 * FG_TILE_FLOATS;
  if (want_sum) sums[tid] = rs;
  __syncthreads();
  if constexpr (!CUT) {
    if (p.c_vec) dg_finish<FG_N, 8, 4, 1>(p, fg_smem, 1, 0, FG_M, m0, n0);
    else dg_finish<FG_N, 8, 1, 4>(p, fg_smem, 1, 0, FG_M, m0, n0);
    if (want_sum && tid < FG_M && m0 + tid < p.M) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += sums[w * 32 + tid];
      p.row_sum[m0 + tid] += v;
    }
  } else {
    float *tot = fg_smem + 8 * FG_TILE_FLOATS;
    {
      const int at = (tid >> 3) * (FG_N + 4) + (tid & 7) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 8; ++w) add4(v, *reinterpret_cast<const float4 *>(fg_smem + w * FG_TILE_FLOATS + at));
      *reinterpret_cast<float4 *>(tot + at) = v;
    }
    if (want_sum && tid < FG_M) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += sums[w * 32 + tid];
      sums[8 * FG_M + tid] = v;
    }
    ptx::cluster_sync_all();
    const int my_rows = FG_M / static_cast<int>(S), first = static_cast<int>(rank) * my_rows;
    if (p.c_vec) dg_finish<FG_N, 1, 4, 1>(p, tot, S, first, my_rows, m0, n0);
    else dg_finish<FG_N, 1, 1, 4>(p, tot, S, first, my_rows, m0, n0);
    if (want_sum && tid < my_rows && m0 + first + tid < p.M) {
      float v = 0.f;
      for (uint32_t q = 0; q < S; ++q) {
        float x;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(ptx::map_to_cta(ptx::smem_u32(sums + 8 * FG_M + first + tid), q)) : "memory");
        v += x;
      }
      p.row_sum[m0 + first + tid] += v;
    }
    ptx::cluster_sync_all();   // a peer may still be reading this CTA's tile
  }
}

// ---------------------------------------------------------------------------------------------------------
// Products whose tiles of 32 x 32 leave most of the chip idle, with plain FMAs on tiles of 16 x 16: four times as many CTAs, a
// quarter of the multiplying each, and twice the operand traffic, which comes from L2.  What remains is latency: all loads of up to
// 256 of K (two chunks) are in flight together whatever the alignment, the third and later chunks travel while one is multiplied,
// and what the epilogue reads is on its way beside them.  (128 x 256 x 256 4.0 us in a chain of launches where 32 x 32 takes 6.2; 203 x
// 333 x 333, rows that are not aligned, 6.8 and 10; a launch without work 3.)  The 8 warps walk interleaved groups of four K and
// their partial tiles are added in warp order (bitwise repeatable).
// ---------------------------------------------------------------------------------------------------------
constexpr int SG_TILE = 16, SG_K = 128, SG_PITCH = SG_K + 4;   // K of a chunk, pitch of an operand's rows in shared memory
constexpr int SG_SMEM = 2 * 2 * SG_TILE * SG_PITCH * 4;          // two chunks; the partial tiles and row sums lie over them
static_assert(SG_SMEM >= (8 * SG_TILE * (SG_TILE + 4) + 8 * SG_TILE) * 4, "the partial tiles lie over the operands");

// The epilogue of a tile of 16 x 16: a thread has VEC adjacent columns of one row at most, summed by `sum(row, column, v)`.  What
// the epilogue reads from memory is on its way before `work`, which computes the partial tiles and ends with them visible to every thread.
// (dg_finish, where a thread has several rows, in this form is slower by 1 to 3 us: 512 x 709 x 64 8.5 -> 10.7.)
template <int VEC, typename Work, typename Sum>
__device__ __forceinline__ void sg_finish(const DirectProblem &p, int m0, int n0, Work work, Sum sum) {
  constexpr int LANES = SG_TILE / VEC;
  using Vec = float[VEC];
  const Epilogue &e = p.epi;
  const int c = (static_cast<int>(threadIdx.x) % LANES) * VEC, n = n0 + c, r = static_cast<int>(threadIdx.x) / LANES;
  const long long m = m0 + r;
  const bool in = n < p.N && r < SG_TILE && m < p.M;
  Vec bias = {}, factor = {}, add = {}, slope, old;   // slope: activation derivative; old: what lies in C
  if (in) {
    if (e.bias != nullptr) ld_cols(bias, e.bias + n);
    if (e.act_out != nullptr) dg_factors<VEC>(e, n, factor);
    if (e.addend != nullptr) ld_cols(add, e.addend + m * e.ld_addend + n);
    if (e.accumulate) ld_cols(old, e.C + c_row(e, m) + n);
    if (e.deriv_af != 0u) {
      float pre[1][VEC], y[1][VEC];
      Vec cs, ch = {};
#pragma unroll
      for (int k = 0; k < VEC; ++k) cs[k] = 1.f;
      if (e.aux_pre != nullptr) ld_cols(pre[0], e.aux_pre + m * e.ld_aux + n);
      if (e.aux_y != nullptr) ld_cols(y[0], e.aux_y + m * e.ld_aux + n);
      if (e.aux_pre != nullptr && e.col_scale != nullptr) { ld_cols(cs, e.col_scale + n); ld_cols(ch, e.col_shift + n); }
      dg_derive<1, VEC>(e, pre, y, cs, ch, [&](int, int k, float x) { slope[k] = x; });
    }
  }
  work();
  if (!in) return;
  float v[1][VEC] = {};
  sum(r, c, v[0]);
#pragma unroll
  for (int k = 0; k < VEC; ++k) {
    v[0][k] += bias[k];
    if (e.addend != nullptr) v[0][k] += add[k];
    if (e.deriv_af != 0u) v[0][k] *= slope[k];
    if (e.accumulate) v[0][k] += old[k];
  }
  st_cols(e.C + c_row(e, m) + n, v[0]);
  if (e.act_out != nullptr) {
    dg_fire<1, VEC>(e, v, factor);
    st_cols(e.act_out + c_row(e, m) + n, v[0]);
  }
}

// One operand's share of a chunk of K on its way from memory through a thread's registers into shared memory: all loads of a chunk
// are in flight together, whatever the alignment.  Rows row0 .. row0 + ROWS - 1 (past `rows`: the last one again), K elements
// k0 .. k0 + kc - 1 (zeros up to a multiple of 4).
template <bool T, int ROWS>
struct SgOperand {
  static constexpr int N = ROWS / 8;   // 16-byte pieces per thread
  const float *src;
  long long ld;
  int row0, rows;
  bool vec;
  struct Set { float4 v[N]; int shift[N]; };

  __device__ __forceinline__ bool wide() const { return vec && row0 + ROWS <= rows; }
  __device__ __forceinline__ void load(Set &x, int k0, int kc) const {
    const int tid = static_cast<int>(threadIdx.x);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (T) {
      if (wide()) {   // lanes take consecutive 16 bytes along the rows
        constexpr int L = ROWS / 4;
        const float *q = src + static_cast<long long>(k0) * ld + row0 + (tid % L) * 4;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int k = tid / L + i * (DG_THREADS / L);
          x.v[i] = k < kc ? *reinterpret_cast<const float4 *>(q + k * ld) : zero;
        }
      } else {
        const float *q = src + static_cast<long long>(k0) * ld + min(row0 + tid % ROWS, rows - 1);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          float e[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = tid / ROWS + (4 * i + j) * (DG_THREADS / ROWS);
            e[j] = k < kc ? q[k * ld] : 0.f;
          }
          x.v[i] = make_float4(e[0], e[1], e[2], e[3]);
        }
      }
    } else {
      // a warp takes a row, its lanes consecutive 16 bytes; a row that does not start on such a boundary is read from the boundary
      // before it, and store() moves the elements to their places
      const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float *q = src + static_cast<long long>(min(row0 + warp + 8 * i, rows - 1)) * ld + k0;
        x.shift[i] = static_cast<int>(reinterpret_cast<uintptr_t>(q) >> 2) & 3;
        const int k = 4 * lane - x.shift[i];
        if (k >= 0 && k + 4 <= kc) {
          x.v[i] = *reinterpret_cast<const float4 *>(q + k);
        } else {
          x.v[i].x = k >= 0 && k < kc ? q[k] : 0.f;
          x.v[i].y = k + 1 >= 0 && k + 1 < kc ? q[k + 1] : 0.f;
          x.v[i].z = k + 2 >= 0 && k + 2 < kc ? q[k + 2] : 0.f;
          x.v[i].w = k + 3 < kc ? q[k + 3] : 0.f;   // (the shift is 3 at most)
        }
      }
    }
  }
  __device__ __forceinline__ void store(const Set &x, float *s, int kc) const {
    const int tid = static_cast<int>(threadIdx.x), kz = (kc + 3) & ~3;
    if constexpr (T) {
      if (wide()) {
        constexpr int L = ROWS / 4;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int k = tid / L + i * (DG_THREADS / L);
          if (k < kz) *reinterpret_cast<float4 *>(s + k * ROWS + (tid % L) * 4) = x.v[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const float e[4] = {x.v[i].x, x.v[i].y, x.v[i].z, x.v[i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = tid / ROWS + (4 * i + j) * (DG_THREADS / ROWS);
            if (k < kz) s[k * ROWS + tid % ROWS] = e[j];
          }
        }
      }
    } else {
      const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        float4 v = x.v[i];
        if (!vec) {
          const float a = __shfl_down_sync(0xffffffffu, v.x, 1), b = __shfl_down_sync(0xffffffffu, v.y, 1), c = __shfl_down_sync(0xffffffffu, v.z, 1);
          if (x.shift[i] == 1) v = make_float4(v.y, v.z, v.w, a);
          else if (x.shift[i] == 2) v = make_float4(v.z, v.w, a, b);
          else if (x.shift[i] == 3) v = make_float4(v.w, a, b, c);
        }
        if (4 * lane < kz) *reinterpret_cast<float4 *>(s + (warp + 8 * i) * SG_PITCH + 4 * lane) = v;
      }
    }
  }
};

template <bool AT, bool BT, int MAX>
__global__ void __launch_bounds__(DG_THREADS, 2) small_gemm_kernel(const __grid_constant__ DirectGroup<MAX> g, const int chunk) {
  constexpr int TM = SG_TILE, TN = SG_TILE, RG = 4, CG = 8, TILE = TM * (TN + 4), BUFFER = (TM + TN) * SG_PITCH;
  extern __shared__ __align__(16) float sg_smem[];
  const int tile = static_cast<int>(blockIdx.x);
  int pi = 0;
#pragma unroll 1
  while (pi + 1 < g.count && tile >= g.p[pi + 1].first_tile) ++pi;
  const DirectProblem &p = g.p[pi];
  const int tl = tile - p.first_tile;
  const int tm = tl / p.tiles_n, tn = tl - tm * p.tiles_n;
  const int m0 = tm * TM, n0 = tn * TN;
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int rg = lane / CG, cg = lane % CG;   // rows rg + 4 i or 4 rg + i, columns cg + 8 j or 2 cg + j
  const bool want_sum = AT && p.row_sum != nullptr && tn == 0;
  const int chunks = (p.K + chunk - 1) / chunk;
  float *sums = sg_smem + 8 * TILE;
  const SgOperand<AT, TM> oa{p.a, p.lda, m0, p.M, p.a_vec != 0};
  const SgOperand<BT, TN> ob{p.b, p.ldb, n0, p.N, p.b_vec != 0};
  typename SgOperand<AT, TM>::Set a_in[2];
  typename SgOperand<BT, TN>::Set b_in[2];
  grid_dependency_wait();
  grid_dependency_release();
  auto length = [&](int c) { return min(chunk, p.K - c * chunk); };
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (j < chunks) {
      oa.load(a_in[j], j * chunk, length(j));
      ob.load(b_in[j], j * chunk, length(j));
    }
  auto work = [&]() {
    float acc[4][2] = {};
    float rs = 0.f;
#pragma unroll 1
    for (int c0 = 0; c0 < chunks; c0 += 2) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = c0 + j;
        if (c >= chunks) break;
        const int kc = length(c);
        float *sa = sg_smem + j * BUFFER, *sb = sa + TM * SG_PITCH;
        oa.store(a_in[j], sa, kc);
        ob.store(b_in[j], sb, kc);
        __syncthreads();   // (what lay in this buffer had been multiplied by everybody before the last of these)
        if (c + 2 < chunks) {
          oa.load(a_in[j], (c + 2) * chunk, length(c + 2));
          ob.load(b_in[j], (c + 2) * chunk, length(c + 2));
        }
        if (want_sum && lane < TM)
          for (int k = warp; k < kc; k += 8) rs += sa[k * TM + lane];
#pragma unroll 2
        for (int k = warp * 4; k < kc; k += 32) {
          float a[4][4], b[4][2];   // [row][k], [k][column]
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4 *>(AT ? sa + (k + i) * TM + rg * 4 : sa + (rg + RG * i) * SG_PITCH + k);
            if (AT) { a[0][i] = t.x; a[1][i] = t.y; a[2][i] = t.z; a[3][i] = t.w; }
            else { a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w; }
          }
          if constexpr (BT) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 t = *reinterpret_cast<const float2 *>(sb + (k + i) * TN + cg * 2);
              b[i][0] = t.x; b[i][1] = t.y;
            }
          } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const float4 t = *reinterpret_cast<const float4 *>(sb + (cg + CG * q) * SG_PITCH + k);
              b[0][q] = t.x; b[1][q] = t.y; b[2][q] = t.z; b[3][q] = t.w;
            }
          }
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int q = 0; q < 2; ++q) acc[i][q] = fmaf(a[i][kk], b[kk][q], acc[i][q]);
        }
      }
    }
    __syncthreads();   // the operands have been read: the partial tiles take their place
    float *part = sg_smem + warp * TILE;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float *d = part + (AT ? rg * 4 + i : rg + RG * i) * (TN + 4);
#pragma unroll
      for (int q = 0; q < 2; ++q) d[BT ? cg * 2 + q : cg + CG * q] = acc[i][q];
    }
    if (want_sum && lane < TM) sums[warp * TM + lane] = rs;
    __syncthreads();
  };
  auto sum = [&](int r, int c, auto &v) {
    constexpr int VEC = sizeof(v) / sizeof(float);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float *t = sg_smem + w * TILE + r * (TN + 4) + c;
      if constexpr (VEC == 4) {
        const float4 x = *reinterpret_cast<const float4 *>(t);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
      } else {
        v[0] += *t;
      }
    }
  };
  if (p.c_vec) sg_finish<4>(p, m0, n0, work, sum);
  else sg_finish<1>(p, m0, n0, work, sum);
  if (want_sum && tid < TM && m0 + tid < p.M) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += sums[w * TM + tid];
    p.row_sum[m0 + tid] += v;
  }
}

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
// Up to 600 M multiply-adds.  Measured against the panel kernels with their splits (us): 512^3 9.0 / 16.0, 256 x 1024 x 1024 12.1 /
// 24.9, 512 x 2048 x 512 16.7 / 19.1, 1024^3 29.1 / 29.4, 2048 x 1024 x 512 27.4 / 22.7: conversion is repeated by every tile that
// reads an operand, which from there on costs more than the split passes (that several contractions share).
bool direct_gemm_suits(const Context &ctx, long long M, long long N, long long K) {
  return ctx.gemm_engine == 0 && ctx.gemm_bn == 0 && M > 0 && N > 0 && K > 0 && M * N * K <= (600ll << 20);
}

template <bool AT, bool BT, int MAX, bool WIDE>
static int launch_direct_reading(Context &ctx, const DirectGroup<MAX> &g, int tiles, int cluster) {
  auto kernel = direct_gemm_kernel<AT, BT, MAX, WIDE>;
  static std::once_flag flags[64];
  static bool ok[64] = {};
  if (ctx.device < 0 || ctx.device >= 64) return MYEA_E_CUDA;
  std::call_once(flags[ctx.device], [&] { ok[ctx.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_SMEM) == cudaSuccess; });
  if (!ok[ctx.device]) return MYEA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * cluster));
  cfg.blockDim = dim3(DG_THREADS);
  cfg.dynamicSmemBytes = DG_SMEM;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (ctx.dependent_launch && !ctx.profiling) ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  ctx.begin(TC_GEMM);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, g, ctx.d_error_flag);
  ctx.end(TC_GEMM);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// Accesses of whole sectors where every operand read through its rows allows 16 bytes at least.  A kernel that has them beside the
// element-wise reads of other rows is slower at those (us without / with them: 512 x 709 x 1001 24.5 / 24.8, the second operand through
// its columns 22.4 / 23.3; 256 x 1024 x 1001 13.6 / 14.1).  Aligned rows: 64 x 6000 x 256 9.7 / 9.4, 512 x 709 x 784 17.7 / 17.1.  Of a short
// K the reading does not matter, and the product takes the kernel that the next one will, which reads its result: two of them in turn
// fetch their instructions anew (784-1024-1024-10 on 256 rows: 3 us of a step of 165).
template <bool AT, bool BT, int MAX>
static int launch_direct(Context &ctx, const DirectGroup<MAX> &g, int tiles, int cluster) {
  if constexpr (!(AT && BT)) {
    bool rows = true, result = true;
    int longest = 0;
    for (int i = 0; i < g.count; ++i) {
      rows = rows && (AT || g.p[i].a_vec) && (BT || g.p[i].b_vec);
      result = result && g.p[i].c_vec;
      longest = std::max(longest, g.p[i].K);
    }
    if (longest >= 256 ? rows : result) return launch_direct_reading<AT, BT, MAX, true>(ctx, g, tiles, cluster);
  }
  return launch_direct_reading<AT, BT, MAX, false>(ctx, g, tiles, cluster);
}

static bool epilogue_is_vector(const Epilogue &e, long long N) {
  return epilogue_vector_ok(e) && (reinterpret_cast<uintptr_t>(e.act_out) & 15) == 0 && (N & 3) == 0;
}

template <bool AT, bool BT, int MAX, bool CUT>
static int launch_fma_cut(Context &ctx, const DirectGroup<MAX> &g, int tiles, int cluster) {
  auto kernel = fma_gemm_kernel<AT, BT, MAX, CUT>;
  static std::once_flag flags[64];
  static bool ok[64] = {};
  if (ctx.device < 0 || ctx.device >= 64) return MYEA_E_CUDA;
  std::call_once(flags[ctx.device], [&] { ok[ctx.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FG_SMEM) == cudaSuccess; });
  if (!ok[ctx.device]) return MYEA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * cluster));
  cfg.blockDim = dim3(DG_THREADS);
  cfg.dynamicSmemBytes = FG_SMEM;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (ctx.dependent_launch && !ctx.profiling) ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CUT ? 2 : 1;
  ctx.begin(TC_GEMM);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, g);
  ctx.end(TC_GEMM);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

template <bool AT, bool BT, int MAX>
static int launch_fma(Context &ctx, const DirectGroup<MAX> &g, int tiles, int cluster) {
  return cluster > 1 ? launch_fma_cut<AT, BT, MAX, true>(ctx, g, tiles, cluster) : launch_fma_cut<AT, BT, MAX, false>(ctx, g, tiles, 1);
}

template <bool AT, bool BT, int MAX>
static int launch_small(Context &ctx, const DirectGroup<MAX> &g, int tiles) {
  int chunk = SG_K;
  for (int i = 0; i < g.count; ++i)
    if ((!AT && !g.p[i].a_vec) || (!BT && !g.p[i].b_vec)) chunk = SG_K - 4;   // (a row that is read from the boundary before it takes one lane more)
  ctx.begin(TC_GEMM);
  const cudaError_t err = launch_dependent(ctx, small_gemm_kernel<AT, BT, MAX>, dim3(static_cast<unsigned>(tiles)), dim3(DG_THREADS), SG_SMEM, g, chunk);
  ctx.end(TC_GEMM);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

static long long operand_pitch(const Operand &o, bool columns) { return columns ? o.stride_k : o.stride_r; }

// How many CTAs share the K range of a 32 x 32 tile, or tensor-core tiles instead.  One CTA per SM at most: two of them take all
// registers of an SM, so that the next launch cannot set itself up beside them (a 256 x 1024 x 10 product alone took 3.4 us instead
// of 4.6, and the training step around it 5 us more).  Estimates (us) from these measurements of FMAs with 1 / 2 / 4 / 8 CTAs and of
// tensor-core tiles: 128 x 256 x 64 3.4 / 4.6 / 4.8 / 5.7, 5.5; 128 x 256 x 256 5.2 / 5.5 / 5.4 / 6.0, 6.8; 64 x 512 x 512 8.4 / 6.7 / 6.2 /
// 6.4, 8.0; 256 x 10 x 1024 15.2 / 10.2 / 7.3 / 6.5, 11.5; 32 x 64 x 4096 54 / 30 / 17 / 10, 17; 384^3 8.0, 7.8; rows that are not
// 16-byte aligned: 203 x 333 x 75 5.3, 9.8; 203 x 333 x 333 9.5 / 11.5, 9.9; 333 x 333 x 203 6.6 / 8.3, 8.6; 161 x 150 x 2000 33 / 20 / 15 / 13, 12.
// Tiles of 16 x 16 (one CTA each) where they are up to two CTAs per SM.  Estimates from these measurements, beside the others':
// 128 x 256 x 64 3.4, 128 x 256 x 256 4.0, 64 x 512 x 512 5.0, 256 x 256 x 512 6.6 (256 tiles), 256 x 10 x 1024 8.4, 32 x 64 x 4096 26; not aligned:
// 203 x 333 x 75 3.4, 203 x 333 x 333 6.8 (273 tiles), 161 x 150 x 2000 read through its columns 20.6.
struct FmaPlan {
  int tile = 0, cluster = 1;   // tile 0: tensor-core tiles
};
static FmaPlan fma_plan(const DirectItem *items, int n, bool at, bool bt) {
  auto tiles_of = [&](long long t) {
    long long tiles = 0;
    for (int i = 0; i < n; ++i) tiles += (items[i].A.rows + t - 1) / t * ((items[i].B.rows + t - 1) / t);
    return tiles;
  };
  long long longest = 0;
  bool aligned = true;
  for (int i = 0; i < n; ++i) {
    longest = std::max(longest, items[i].A.k);
    aligned = aligned && ((reinterpret_cast<uintptr_t>(items[i].A.ptr) | reinterpret_cast<uintptr_t>(items[i].B.ptr)) & 15) == 0 &&
              ((operand_pitch(items[i].A, at) | operand_pitch(items[i].B, bt)) & 3) == 0;
  }
  const double K = static_cast<double>(longest);
  double best = 5.0 + 0.006 * std::min(K, 1024.0) + 0.002 * std::max(0.0, K - 1024.0) + (aligned ? 0.0 : 2.0) - 0.5;
  FmaPlan plan;
  const long long t32 = tiles_of(FG_M), t16 = tiles_of(SG_TILE);
  // (rows off the 16-byte boundaries take tiles of 32 x 32 about twice as long per K.  That decides between the two FMA tiles; against
  // the tensor-core tiles, which are hardly faster there and less exact, it does not count)
  double fma = 1e30;
  for (int S = 1; S <= 8 && t32 * S <= 148; S *= 2) {
    const double walk = 0.011 * K / S, t = 2.6 + walk + (S > 1 ? 2.2 : 0.0) + (S == 8 ? 0.5 : 0.0);
    if (t < best) { best = t; fma = t + (aligned ? 0.0 : walk); plan.tile = FG_M; plan.cluster = S; }
  }
  if (t16 <= 296 && 2.4 + 0.0055 * K * (t16 > 148 ? 1.6 : 1.0) * (aligned ? 1.0 : 1.5) < (plan.tile ? fma : best)) {
    plan.tile = SG_TILE;
    plan.cluster = 1;
  }
  return plan;
}

// How the operands of a launch are read: through their columns (rows contiguous, pitch stride_k) or their rows (K contiguous,
// pitch stride_r).  All items share the choice, and an operand of a single row or a single K can be read either way whatever
// its strides say: the errors of a layer of one unit are a column of pitch 1, which beside wider layers is read as theirs are.
static bool reads_columns(const Operand &o) { return o.stride_r == 1 || o.rows == 1; }
static bool reads_rows(const Operand &o) { return o.stride_k == 1 || o.k == 1; }
static bool choose_reading(const DirectItem *items, int n, Operand DirectItem::*which, bool columns, bool *out) {
  bool all_columns = true, all_rows = true;
  for (int i = 0; i < n; ++i) {
    const Operand &o = items[i].*which;
    columns = columns || o.stride_k != 1;
    all_columns = all_columns && reads_columns(o);
    all_rows = all_rows && reads_rows(o);
  }
  *out = columns && all_columns;
  return *out || all_rows;
}

// How a launch runs: readings of its operands, tile and CTAs per tile
struct DirectPlan {
  bool at = false, bt = false;
  int tile_m = DG_M, tile_n = DG_N, cluster = 1;
};
static bool plan_direct(const DirectItem *items, int n, DirectPlan *plan) {
  bool sums = false;
  for (int i = 0; i < n; ++i) sums = sums || items[i].row_sum != nullptr;   // these are taken from operands read through their columns
  if (!choose_reading(items, n, &DirectItem::A, sums, &plan->at) || !choose_reading(items, n, &DirectItem::B, false, &plan->bt)) return false;
  const FmaPlan fma = fma_plan(items, n, plan->at, plan->bt);
  if (fma.tile != 0) {
    plan->tile_m = plan->tile_n = fma.tile;
    plan->cluster = fma.cluster;
    return true;
  }
  long long tiles = 0, min_steps = 1 << 30;
  for (int i = 0; i < n; ++i) {
    tiles += (items[i].A.rows + DG_M - 1) / DG_M * ((items[i].B.rows + DG_N - 1) / DG_N);
    min_steps = std::min(min_steps, (items[i].A.k + BK - 1) / BK);
  }
  // K is cut in up to four while the grid stays within one CTA per SM and every CTA keeps two stages.  Measured (us per
  // launch, cut 1 / 2 / 4 / 8): 128 x 256 x 256 9.6 / 8.0 / 6.6 / 7.2, 203 x 333 x 333 18.6 / 13.6 / 9.8 / 11.3, 512^3 15.7 / 11.2
  // / 8.8 / 12.3, 640^3 18.7 / 12.8 / 13.1 / 24.3, 1024 x 1024 x 256 10.1 / 11.1 / 18.0: clusters of eight are placed late, and
  // pay only for very long walks (64 x 2048 x 2048: 53.0 / 30.1 / 17.8 / 16.6)
  int &cluster = plan->cluster;
  while (cluster < (min_steps >= 64 ? 8 : 4) && tiles * cluster * 2 <= (cluster == 4 ? 256 : 148) && min_steps >= cluster * 4) cluster *= 2;
  return true;
}

template <bool AT, bool BT, int MAX>
static int launch_planned(Context &ctx, const DirectGroup<MAX> &g, int tiles, const DirectPlan &plan) {
  if (plan.tile_m == SG_TILE) return launch_small<AT, BT, MAX>(ctx, g, tiles);
  if (plan.tile_m == FG_M) return launch_fma<AT, BT, MAX>(ctx, g, tiles, plan.cluster);
  return launch_direct<AT, BT, MAX>(ctx, g, tiles, plan.cluster);
}

template <int MAX>
static int direct_gemm_launch(Context &ctx, const DirectItem *items, int n) {
  DirectGroup<MAX> g;
  g.count = n;
  int tiles = 0;
  DirectPlan plan;
  if (!plan_direct(items, n, &plan)) return MYEA_E_INVALID;
  const bool at = plan.at, bt = plan.bt;
  for (int i = 0; i < n; ++i) {
    const DirectItem &it = items[i];
    DirectProblem &p = g.p[i];
    if (it.A.k != it.B.k || it.A.rows <= 0 || it.B.rows <= 0 || it.A.k <= 0) return MYEA_E_INVALID;
    p.a = it.A.ptr; p.b = it.B.ptr;
    p.lda = operand_pitch(it.A, at);
    p.ldb = operand_pitch(it.B, bt);
    p.M = static_cast<int>(it.A.rows); p.N = static_cast<int>(it.B.rows); p.K = static_cast<int>(it.A.k);
    p.a_vec = (reinterpret_cast<uintptr_t>(p.a) & 15) == 0 && (p.lda & 3) == 0;
    p.b_vec = (reinterpret_cast<uintptr_t>(p.b) & 15) == 0 && (p.ldb & 3) == 0;
    p.c_vec = epilogue_is_vector(it.epi, p.N);
    p.tiles_n = (p.N + plan.tile_n - 1) / plan.tile_n;
    p.first_tile = tiles;
    tiles += p.tiles_n * ((p.M + plan.tile_m - 1) / plan.tile_m);
    p.row_sum = at ? it.row_sum : nullptr;
    p.epi = it.epi;
    if ((it.row_sum != nullptr && !at) || it.epi.stats_kind != 0) return MYEA_E_INVALID;
    ctx.gemm_flops += 2.0 * p.M * p.N * static_cast<double>(p.K);
  }
  if (at) return bt ? launch_planned<true, true>(ctx, g, tiles, plan) : launch_planned<true, false>(ctx, g, tiles, plan);
  return bt ? launch_planned<false, true>(ctx, g, tiles, plan) : launch_planned<false, false>(ctx, g, tiles, plan);
}

// Items of one call are read alike: all A through their rows or all through their columns, and all B.
int direct_gemm(Context &ctx, const DirectItem *items, int count) {
  for (int first = 0; first < count; first += DG_MAX_ITEMS) {
    const int n = std::min(DG_MAX_ITEMS, count - first);
    const int rc = n == 1 ? direct_gemm_launch<1>(ctx, items + first, n) : direct_gemm_launch<DG_MAX_ITEMS>(ctx, items + first, n);
    if (rc != MYEA_OK) return rc;
  }
  return MYEA_OK;
}

}  // namespace myea

// For tests: how a product [M, K] x [N, K]^T of operands that start on 16-byte boundaries runs; columns: bit 0 / 1, A / B is read through its columns.
// tile: rows of a tile, 16 and 32 with FMAs, 128 on the tensor cores straight from fp32, 256 from operand panels; ctas: that share a tile (0 for panels).
extern "C" int myea_b200_contraction_plan(uint64_t M, uint64_t N, uint64_t K, int columns, int *tile, int *ctas) {
  if (M == 0 || N == 0 || K == 0 || tile == nullptr || ctas == nullptr) return MYEA_E_INVALID;
  const long long m = static_cast<long long>(M), n = static_cast<long long>(N), k = static_cast<long long>(K);
  *tile = 256;
  *ctas = 0;
  if (!myea::direct_gemm_suits(myea::Context(), m, n, k)) return MYEA_OK;
  myea::DirectItem item;
  item.A = (columns & 1) != 0 ? myea::Operand{nullptr, m, k, 1, m} : myea::Operand{nullptr, m, k, k, 1};
  item.B = (columns & 2) != 0 ? myea::Operand{nullptr, n, k, 1, n} : myea::Operand{nullptr, n, k, k, 1};
  myea::DirectPlan plan;
  if (!myea::plan_direct(&item, 1, &plan)) return MYEA_E_INVALID;
  *tile = plan.tile_m;
  *ctas = plan.cluster;
  return MYEA_OK;
}
