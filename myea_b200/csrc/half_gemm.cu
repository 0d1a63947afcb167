// Dense contractions of the training step on Blackwell tensor cores.
//
//   C[M,N] (+)= A[M,K] * B[N,K]^T        fp32 in, fp32 out
//
// replaces the three scalar triple loops of the reference: Forward_Pass__FC
// (Neural_Network__Forward_Pass__OpenMP.cpp:4517-4557), Backward_Pass__FC (…Backward_Pass__OpenMP.cpp:1044-1082) and
// Update_Derivative_Weight__FC (…Update_Derivative_Weight__OpenMP.cpp:178-216), and the LSTM gate products.
//
// Operands come as half panels (half_panels.cuh): x = (h0 + h1) * 2^e.  Per 16 of K three tcgen05.mma kind::f16
// (h1*h0, h0*h1, h0*h0) accumulate in fp32 in tensor memory.  An exponent belongs to one row of an operand and 128 of K, and an
// accumulator holds 128 of K: the drain multiplies it by the powers of two of its row and column while it adds it to the running
// sum.
//
// One kernel, persistent: a CTA pair (cta_group::2) computes 256 x BN output tiles (BN = 256; 128 where N <= 128), each
// CTA 128 rows.  384 threads in three warpgroups:
//   warp 0      TMA producer: per stage 64 of K, 128 rows of A and BN / 2 rows of B, both halves (64 KB, 3 stages)
//   warp 1      one lane of the leader CTA issues the twelve tcgen05.mma of a stage; tcgen05.commit releases the stage on both CTAs
//   warps 4-11  drain: tensor memory holds two accumulators; all products of one chunk (2 stages = 128 of K, 24
//               instructions) go into one while the eight drain warps add the other, scaled, to fp32 registers.  A chain
//               of truncating tensor-core adds is never longer than 24 instructions, whatever K is.
// The roles keep running stage / chunk counters across tiles, so the loads and products of the next tile start while the
// drain warps, which hold the finished tile in registers, run its epilogue.  setmaxnreg moves the registers of the role
// warps to the drain warps.  Tiles are numbered in bands of 8 row tiles so that the tiles in flight share operand panels
// in L2.  Every mbarrier wait is bounded (about one second of SM clock); a wait that runs out sets the handle's error
// flag and the CTA pair frees its tensor memory and returns.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "half_panels.cuh"
#include "panel_math.cuh"
#include "tcgen05.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

namespace myea {

struct GemmDims {
  int M, N, K;
};

constexpr int HG_STAGES = 3;
constexpr int HG_THREADS = 384;
constexpr int HG_DRAIN_WARP0 = 4;
constexpr int HG_BK = 64;         // K per stage: 128 bytes of halves
constexpr int HG_KC = 2;          // stages per chunk
constexpr int HG_BAND = 8;
static_assert(HG_BK * HG_KC == HP_BLOCK, "an accumulator covers one exponent block of K");
template <int BN> struct HalfSmem {
  static constexpr int A_BYTES = 128 * 128;                 // 128 rows x 128 bytes
  static constexpr int B_BYTES = BN / 2 * 128;
  static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;  // A h0, A h1, B h0, B h1
  static constexpr int BAR_OFFSET = HG_STAGES * STAGE_BYTES;
  static constexpr int TR_OFFSET = BAR_OFFSET + 512;        // epilogue staging: 8 warps x 32 x 32 floats (the stages stay busy)
  static constexpr int TOTAL = TR_OFFSET + 8 * TR_WARP_FLOATS * 4 + 1024;
};

// Work list.  Tiles [0, dp_tiles) are computed whole, round-robin over the clusters.  The K chunks of the remaining tiles
// (the partial last wave, or every tile of a contraction with fewer tiles than clusters) form one sequence of sk_units
// chunks that is cut into equal runs of sk_chunks, one run per cluster ("stream-K"), so that the tail of the work list is
// spread over all SM pairs instead of leaving most of them idle.
struct WideWork {
  int tiles_m, tiles_n, num_tiles;
  int dp_tiles;
  int sk_chunks;           // chunks per cluster of the split part (0: nothing is split)
  int sk_units;            // (num_tiles - dp_tiles) * chunks per tile
  float *ws;               // partial sums of split tiles: [cluster][2][16 warp regions][BN / 8 float4 columns][32 lanes]
  unsigned int *counters;  // [split tile][16 warp regions] arrivals; the last arrival adds the partials up and resets it
};
constexpr int HG_REGION_FLOATS = 32 * 128;  // one drain warp's share of a 256 x 256 tile: 32 rows x 128 columns

// powers of two of an operand as the kernel walks them: chunk c of K, block b of 128 of its rows
struct ScaleView {
  const uint16_t *p;
  long long step_k;
  int last;   // blocks past the tensor repeat the last one
  __device__ __forceinline__ const uint16_t *block(int b) const { return p + static_cast<long long>(min(b, last)) * HP_BLOCK; }
};

// two neighbouring columns in packed arithmetic (half the instructions): sum += product * column's power of two * row's
__device__ __forceinline__ void scaled_add2(float &s0, float &s1, uint32_t r0, uint32_t r1, uint32_t columns, uint64_t row) {
  asm("{\n"
      ".reg .b64 r, c, s;\n"
      "mov.b64 r, {%2, %3};\n"
      "mov.b64 c, {%4, %5};\n"
      "mov.b64 s, {%0, %1};\n"
      "mul.rn.f32x2 r, r, c;\n"
      "fma.rn.f32x2 s, r, %6, s;\n"
      "mov.b64 {%0, %1}, s;\n"
      "}\n"
      : "+f"(s0), "+f"(s1)
      : "r"(r0), "r"(r1), "r"(columns << 16), "r"(columns & 0xffff0000u), "l"(row));
}

// What the epilogue will read of one row of a tile, on its way from HBM to L2 while the products are computed: behind the last of
// them a single-wave contraction otherwise waits for arrays that earlier launches have left there.
template <int COLS>
__device__ __forceinline__ void prefetch_epilogue(const Epilogue &e, long long row, long long col, long long M, long long N) {
  if (row >= M) return;
  auto line = [](const float *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); };
#pragma unroll
  for (int j = 0; j < COLS; j += 32) {
    if (col + j >= N) break;
    if (e.aux_pre != nullptr) line(e.aux_pre + row * e.ld_aux + col + j);
    if (e.aux_y != nullptr) line(e.aux_y + row * e.ld_aux + col + j);
    if (e.addend != nullptr) line(e.addend + row * e.ld_addend + col + j);
    if (e.accumulate) line(e.C + c_row(e, row) + col + j);
  }
}

__device__ __forceinline__ void wide_tile_coords(const WideWork &w, int t, int &tm, int &tn) {
  const int per_band = HG_BAND * w.tiles_n;
  const int band = t / per_band;
  const int within = t - band * per_band;
  const int rows = min(HG_BAND, w.tiles_m - band * HG_BAND);
  tn = within / rows;
  tm = band * HG_BAND + (within - tn * rows);
}

// The segments (tile, chunk range) of one cluster, in the order every role of the kernel walks them.
struct WideSegments {
  int next_tile, stride, dp_tiles, num_chunks, u, u_end;
  int tile, c0, c1;  // the current segment
  __device__ __forceinline__ WideSegments(const WideWork &w, int cluster, int clusters, int chunks_per_tile)
      : next_tile(cluster), stride(clusters), dp_tiles(w.dp_tiles), num_chunks(chunks_per_tile) {
    u = min(cluster * w.sk_chunks, w.sk_units);
    u_end = min(u + w.sk_chunks, w.sk_units);
  }
  __device__ __forceinline__ bool next() {
    if (next_tile < dp_tiles) {
      tile = next_tile; c0 = 0; c1 = num_chunks;
      next_tile += stride;
      return true;
    }
    if (u < u_end) {
      const int ts = u / num_chunks;
      c0 = u - ts * num_chunks;
      if (c0 + (u_end - u) > num_chunks) {
        // The run crosses into the next tile (a run is shorter than a tile, so it touches two at most): the head of
        // the next tile goes first and the end of this tile after it.  Every cluster then walks K upwards from chunk 0
        // at the same time as the clusters on the neighbouring tiles, which read the same operand panels, and the
        // panels are fetched from DRAM once instead of once per tile.
        tile = dp_tiles + ts + 1;
        c0 = 0;
        c1 = u_end - (ts + 1) * num_chunks;
        u_end = (ts + 1) * num_chunks;
        return true;
      }
      c1 = min(num_chunks, c0 + (u_end - u));
      tile = dp_tiles + ts;
      u += c1 - c0;
      return true;
    }
    return false;
  }
};

// one operand's ROWS rows of one stage: read through the tensor's rows one 2-D box per half (64 of K x ROWS rows), through
// its columns one 3-D box (64 rows of the operand x 64 of K x ROWS / 64 chunks)
template <bool COLS>
__device__ __forceinline__ void half_load_operand(uint8_t *dst0, uint8_t *dst1, const CUtensorMap *m0, const CUtensorMap *m1, uint64_t *bar, int kb, int row0) {
  if (!COLS) {
    ptx::tma_load_2d_pair(dst0, m0, bar, kb * HG_BK, row0);
    ptx::tma_load_2d_pair(dst1, m1, bar, kb * HG_BK, row0);
  } else {
    ptx::tma_load_3d_pair(dst0, m0, bar, 0, kb * HG_BK, row0 >> 6);
    ptx::tma_load_3d_pair(dst1, m1, bar, 0, kb * HG_BK, row0 >> 6);
  }
}

template <bool COLS>
__device__ __forceinline__ void half_prefetch_operand(const CUtensorMap *m, int kb, int row0) {
  if (!COLS) asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(m), "r"(kb * HG_BK), "r"(row0) : "memory");
  else asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(m), "r"(0), "r"(kb * HG_BK), "r"(row0 >> 6) : "memory");
}

template <int BN, bool A_COLS, bool B_COLS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(HG_THREADS, 1)
half_gemm_kernel(const __grid_constant__ CUtensorMap tm_a0, const __grid_constant__ CUtensorMap tm_a1, const __grid_constant__ CUtensorMap tm_b0,
                 const __grid_constant__ CUtensorMap tm_b1, const ScaleView scale_a, const ScaleView scale_b, const GemmDims dims, const WideWork work,
                 const Epilogue epi, const int variant, int *error_flag) {
  using S = HalfSmem<BN>;
  constexpr int STAGES = HG_STAGES, TMEM_COLS = 2 * BN, HALF_N = BN / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(smem + S::BAR_OFFSET);
  uint64_t *empty_bar = full_bar + STAGES;
  uint64_t *acc_full_bar = empty_bar + STAGES;   // [2] a buffer holds a finished K chunk (multicast to both CTAs)
  uint64_t *acc_empty_bar = acc_full_bar + 2;    // [2] leader only: every drain warp of both CTAs has read the buffer
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(acc_empty_bar + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = ptx::cluster_ctarank();
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;
  const int num_kb = (dims.K + HG_BK - 1) / HG_BK;
  const int num_chunks = (num_kb + HG_KC - 1) / HG_KC;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&acc_full_bar[b], 1);
      ptx::mbar_init(&acc_empty_bar[b], 16);  // one arrival per drain warp of the pair
    }
    *abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_holder, TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  if (warp == 0 && lane == 0) {
    // The first stages' rows of B on their way from HBM to L2 while the launch before this one drains (all CTAs at once want 28 MB
    // before the first product).  A prefetch is no read: what that launch may still write there reaches L2 all the same.
    WideSegments seg(work, cluster_id, num_clusters, num_chunks);
    if (seg.next()) {
      int tm, tn;
      wide_tile_coords(work, seg.tile, tm, tn);
      const int nb0 = tn * BN + static_cast<int>(cta_rank) * HALF_N;
      for (int kb = seg.c0 * HG_KC; kb < min(num_kb, seg.c0 * HG_KC + STAGES); ++kb) {
        half_prefetch_operand<B_COLS>(&tm_b0, kb, nb0);
        half_prefetch_operand<B_COLS>(&tm_b1, kb, nb0);
      }
    }
  }
  grid_dependency_wait();     // everything above read no global memory
  grid_dependency_release();

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    ptx::reg_release<40>();
    if (lane == 0) {
      bool ok = true;
      uint32_t it = 0;  // k-blocks staged so far, over all segments
      WideSegments seg(work, cluster_id, num_clusters, num_chunks);
      while (ok && seg.next()) {
        int tm, tn;
        wide_tile_coords(work, seg.tile, tm, tn);
        const int m0 = tm * 256 + static_cast<int>(cta_rank) * 128;
        const int nb0 = tn * BN + static_cast<int>(cta_rank) * HALF_N;
        const int kb_end = min(num_kb, seg.c1 * HG_KC);
        for (int kb = seg.c0 * HG_KC; kb < kb_end; ++kb, ++it) {
          const int s = static_cast<int>(it % STAGES);
          const uint32_t ph = (it / STAGES) & 1u;
          if (!ptx::mbar_wait_or_abort(&empty_bar[s], ph ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t *st = smem + s * S::STAGE_BYTES;
          if (cta_rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], 2 * S::STAGE_BYTES);
          half_load_operand<A_COLS>(st, st + S::A_BYTES, &tm_a0, &tm_a1, &full_bar[s], kb, m0);
          half_load_operand<B_COLS>(st + 2 * S::A_BYTES, st + 2 * S::A_BYTES + S::B_BYTES, &tm_b0, &tm_b1, &full_bar[s], kb, nb0);
        }
      }
      if (!ok) atomicCAS(error_flag, 0, 301);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA) ----------------
    ptx::reg_release<40>();
    if (lane == 0 && cta_rank == 0) {
      bool ok = true;
      constexpr uint32_t idesc = make_idesc_f16(256, BN, A_COLS, B_COLS);
      // descriptor advance per 16 of K (in 16-byte units): 32 bytes inside the swizzle row of a tile read through its rows,
      // two atoms of 8 K rows of one read through its columns
      constexpr uint64_t a_step = A_COLS ? 128 : 2, b_step = B_COLS ? 128 : 2;
      uint32_t it = 0;  // k-blocks consumed so far
      uint32_t g = 0;   // K chunks issued so far: chunk g goes into buffer g & 1
      // the barriers of the next K block are asked before this one's instructions are issued: while the tensor core reads its
      // operands a look at shared memory takes hundreds of cycles, which would drain the short instruction queue
      bool full_ok = false, acc_ok = false;
      WideSegments seg(work, cluster_id, num_clusters, num_chunks);
      while (ok && seg.next()) {
        for (int c = seg.c0; c < seg.c1 && ok; ++c, ++g) {
          const uint32_t b = g & 1u;
          if (g >= 2) {
            if (!acc_ok && !ptx::mbar_wait_or_abort(&acc_empty_bar[b], ((g >> 1) - 1u) & 1u, abort_flag)) { ok = false; break; }
            ptx::tc_fence_after();
          }
          acc_ok = false;
          const uint32_t acc = tmem_base + b * static_cast<uint32_t>(BN);
          const int kb_end = min(num_kb, (c + 1) * HG_KC);
          for (int kb = c * HG_KC; kb < kb_end; ++kb, ++it) {
            const int s = static_cast<int>(it % STAGES);
            const uint32_t ph = (it / STAGES) & 1u;
            if (!full_ok && !ptx::mbar_wait_or_abort(&full_bar[s], ph, abort_flag)) { ok = false; break; }
            ptx::tc_fence_after();
            full_ok = ptx::mbar_test(&full_bar[(it + 1) % STAGES], ((it + 1) / STAGES) & 1u);
            if (kb + 1 == kb_end && g >= 1) acc_ok = ptx::mbar_test(&acc_empty_bar[b ^ 1u], (((g + 1) >> 1) - 1u) & 1u);
            const uint32_t st = ptx::smem_u32(smem + s * S::STAGE_BYTES);
            const uint32_t sb = st + 2 * S::A_BYTES;
            const uint64_t a0 = A_COLS ? make_smem_desc_mn(st, 8192, false) : make_smem_desc(st);
            const uint64_t a1 = A_COLS ? make_smem_desc_mn(st + S::A_BYTES, 8192, false) : make_smem_desc(st + S::A_BYTES);
            const uint64_t b0 = B_COLS ? make_smem_desc_mn(sb, 8192, false) : make_smem_desc(sb);
            const uint64_t b1 = B_COLS ? make_smem_desc_mn(sb + S::B_BYTES, 8192, false) : make_smem_desc(sb + S::B_BYTES);
#pragma unroll
            for (int k = 0; k < HG_BK / 16; ++k) {
              const bool first = (kb == c * HG_KC) && (k == 0);
              ptx::mma_bf16_pair(acc, a1 + k * a_step, b0 + k * b_step, idesc, first ? 0u : 1u);
              ptx::mma_bf16_pair(acc, a0 + k * a_step, b1 + k * b_step, idesc, 1u);
              ptx::mma_bf16_pair(acc, a0 + k * a_step, b0 + k * b_step, idesc, 1u);
            }
            ptx::tc_commit_pair(&empty_bar[s]);
          }
          if (ok) ptx::tc_commit_pair(&acc_full_bar[b]);
        }
      }
      if (!ok) atomicCAS(error_flag, 0, 302);
    }
  } else if (warp >= HG_DRAIN_WARP0) {
    // ---------------- drain + epilogue: 8 warps; lane quarter = warp % 4, column half = (warp - 4) / 4 ----------------
    ptx::reg_acquire<232>();
    const int q = warp & 3;
    const int half = (warp - HG_DRAIN_WARP0) >> 2;
    const int region = static_cast<int>(cta_rank) * 8 + (warp - HG_DRAIN_WARP0);  // this warp's 32 x HALF_N share of the pair's tile
    float *tr = reinterpret_cast<float *>(smem + S::TR_OFFSET) + (warp - HG_DRAIN_WARP0) * TR_WARP_FLOATS;
    bool ok = true;
    uint32_t g = 0;
    WideSegments seg(work, cluster_id, num_clusters, num_chunks);
    while (ok && seg.next()) {
      int tm, tn;
      wide_tile_coords(work, seg.tile, tm, tn);
      const uint16_t *pa = scale_a.block(tm * 2 + static_cast<int>(cta_rank)) + q * 32 + lane;
      const uint16_t *pb = scale_b.block((tn * BN + half * HALF_N) / HP_BLOCK) + (half * HALF_N) % HP_BLOCK;
      prefetch_epilogue<HALF_N>(epi, static_cast<long long>(tm) * 256 + static_cast<long long>(cta_rank) * 128 + q * 32 + lane,
                                static_cast<long long>(tn) * BN + half * HALF_N, dims.M, dims.N);
      float sum[HALF_N];
#pragma unroll
      for (int j = 0; j < HALF_N; ++j) sum[j] = 0.f;
      for (int c = seg.c0; c < seg.c1; ++c, ++g) {
        const uint32_t b = g & 1u;
        // Powers of two of this lane's row and of the columns (32 of them ahead of the products they belong to).  The column's
        // comes first, times 2^-14 as it is kept, and the row's times 2^14 after it, so that the step between leaves the range
        // of fp32 only for columns beyond 2^118.
        const uint32_t row_bits = (static_cast<uint32_t>(pa[c * scale_a.step_k]) << 16) + (28u << 23);
        const uint64_t sa = static_cast<uint64_t>(row_bits) << 32 | row_bits;
        const uint4 *sb = reinterpret_cast<const uint4 *>(pb + c * scale_b.step_k);
        uint4 next[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) next[i] = sb[i];
        if (!ptx::mbar_wait_or_abort(&acc_full_bar[b], (g >> 1) & 1u, abort_flag)) {
          ok = false;
          if (lane == 0) atomicCAS(error_flag, 0, 303);
          break;
        }
        ptx::tc_fence_after();
        const uint32_t tsrc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + b * static_cast<uint32_t>(BN) + static_cast<uint32_t>(half * HALF_N);
#pragma unroll
        for (int jc = 0; jc < HALF_N / 32; ++jc) {
          uint32_t r[32];
          ptx::tmem_ld_32x32(tsrc + static_cast<uint32_t>(jc * 32), r);
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            w[4 * i] = next[i].x; w[4 * i + 1] = next[i].y; w[4 * i + 2] = next[i].z; w[4 * i + 3] = next[i].w;
            if (jc + 1 < HALF_N / 32) next[i] = sb[4 * (jc + 1) + i];
          }
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            scaled_add2(sum[jc * 32 + j], sum[jc * 32 + j + 1], r[j], r[j + 1], w[j / 2], sa);
          }
        }
        // this warp's reads of the buffer are complete: hand it back to the MMA issuer
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(&acc_empty_bar[b], 0);
      }
      if (!ok || num_kb <= 0) break;
      bool finish = true;  // this warp writes its share of the tile
      if (seg.c0 != 0 || seg.c1 != num_chunks) {
        // A split tile.  Every contributor leaves its partial sums in its own slot and counts itself in; the warp that
        // arrives last adds the slots up in cluster order (the same order whoever is last, so the result does not
        // depend on timing) and runs the epilogue.  Nobody waits for anybody.
        const int ts = seg.tile - work.dp_tiles;
        const int tile_u0 = ts * num_chunks;
        const int first = tile_u0 / work.sk_chunks;
        const int last = min((tile_u0 + num_chunks - 1) / work.sk_chunks, num_clusters - 1);
        auto slot_of = [&](int cluster) {
          const int slot = (cluster * work.sk_chunks >= tile_u0) ? 0 : 1;
          return reinterpret_cast<float4 *>(work.ws + (static_cast<size_t>(cluster * 2 + slot) * 16 + region) * HG_REGION_FLOATS);
        };
        float4 *mine = slot_of(cluster_id);
#pragma unroll
        for (int j = 0; j < HALF_N / 4; ++j) __stcg(mine + j * 32 + lane, make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]));
        __threadfence();
        __syncwarp();
        unsigned int arrived = 0;
        unsigned int *counter = work.counters + ts * 16 + region;
        if (lane == 0) arrived = atomicAdd(counter, 1u);
        arrived = __shfl_sync(0xffffffffu, arrived, 0);
        finish = arrived == static_cast<unsigned int>(last - first);
        if (finish) {
          if (lane == 0) *counter = 0u;  // every contributor has arrived: ready for the next launch
          __threadfence();
          const bool two = last == first + 1;
          // two contributors (the usual case): a + b is the same whichever of them is last, so the sum in registers stays
          // and only the other slot is read; more: every slot is added from zero in cluster order
          if (!two) {
#pragma unroll
            for (int j = 0; j < HALF_N; ++j) sum[j] = 0.f;
          }
#pragma unroll 1
          for (int cc = first; cc <= last; ++cc) {
            if (two && cc == cluster_id) continue;
            const float4 *theirs = slot_of(cc);
#pragma unroll
            for (int jb = 0; jb < HALF_N / 4; jb += 16) {
              float4 v[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __ldcg(theirs + (jb + j) * 32 + lane);
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                sum[4 * (jb + j)] += v[j].x; sum[4 * (jb + j) + 1] += v[j].y; sum[4 * (jb + j) + 2] += v[j].z; sum[4 * (jb + j) + 3] += v[j].w;
              }
            }
          }
        }
      }
      if (finish) {
        const long long row0 = static_cast<long long>(tm) * 256 + static_cast<long long>(cta_rank) * 128 + q * 32;
        epilogue_strip<HALF_N>(epi, variant, tr, sum, lane, row0, static_cast<long long>(tn) * BN + half * HALF_N, dims.M, dims.N);
      }
    }
  } else {
    ptx::reg_release<40>();  // warps 2-3: no role, but the whole warpgroup has to give its registers back
  }
  // every role leaves its loop only when its segments are done or a wait has given up; the pair stays together until
  // both CTAs are here, so nobody signals a barrier of a CTA that has exited
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// fp32 -> panels
struct SplitSource {
  const float *src;
  long long stride;
  RowSegments seg;
  bool vec;
  struct Cols {};
  __device__ __forceinline__ void columns(Cols &, long long, int) const {}
  __device__ __forceinline__ void row(const Cols &, long long r, long long c, int n, float (&v)[8]) const {
    const float *s = src;
    if (seg.seg_rows == 0) {
      s += r * stride;
    } else {
      const int g = static_cast<int>(r >= seg.seg_rows) + static_cast<int>(r >= 2 * seg.seg_rows) + static_cast<int>(r >= 3 * seg.seg_rows);
      s += (r - g * seg.seg_rows) * stride + seg.seg_off[g];
    }
    ld8(v, s + c, n, vec);
  }
  __device__ __forceinline__ void keep(long long, long long, int, const float (&)[8]) const {}
};

// ---------------------------------------------------------------------------------------------------------
// FP32 FMA engine: 64x64 tile, 16 of K per step, 256 threads x (4x4) outputs, arbitrary strides
// ---------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gemm_fp32_fma_kernel(const Operand A, const Operand B, const GemmDims dims, const Epilogue epi) {
  __shared__ float sa[16][64 + 4];
  __shared__ float sb[16][64 + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const long long m0 = static_cast<long long>(blockIdx.y) * 64, n0 = static_cast<long long>(blockIdx.x) * 64;
  float acc[4][4] = {};
  for (long long k0 = 0; k0 < dims.K; k0 += 16) {
    for (int i = threadIdx.x; i < 64 * 16; i += 256) {
      int r, kk;
      if (A.stride_k == 1) { r = i >> 4; kk = i & 15; } else { kk = i >> 6; r = i & 63; }
      const long long m = m0 + r, k = k0 + kk;
      sa[kk][r] = (m < dims.M && k < dims.K) ? A.ptr[m * A.stride_r + k * A.stride_k] : 0.f;
      if (B.stride_k == 1) { r = i >> 4; kk = i & 15; } else { kk = i >> 6; r = i & 63; }
      const long long n = n0 + r;
      sb[kk][r] = (n < dims.N && k0 + kk < dims.K) ? B.ptr[n * B.stride_r + (k0 + kk) * B.stride_k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = sa[kk][ty * 4 + i]; b[i] = sb[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      if (m < dims.M && n < dims.N) epi.C[c_row(epi, m) + n] = epilogue_value<true>(epi, acc[i][j], m, n);
    }
}

// ---------------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  // function-local static: initialised once, by one thread, before any caller sees the pointer
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
  }();
  return fn;
}

// First-use set-up per (kernel, device): the opt-in to large dynamic shared memory is a per-device attribute of the
// kernel.  One table per kernel, indexed by the full device number and guarded, so that two host threads that drive
// two GPUs can make their first calls at the same time.
constexpr int kMaxDevices = 64;
struct PerDeviceOnce {
  std::mutex mutex;
  int value[kMaxDevices] = {};  // 0 = not configured yet
  // returns the cached value (> 0) or the result of `configure` (<= 0 on failure, not cached)
  template <typename F> int get(int device, F configure) {
    if (device < 0 || device >= kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(mutex);
    if (value[device] == 0) {
      const int v = configure();
      if (v > 0) value[device] = v;
      return v;
    }
    return value[device];
  }
};

// map of one half array of an operand: boxes of 64 of K x `box_rows` operand rows, 128-byte swizzle; what lies outside the
// operand is filled with zeros
bool make_half_map(CUtensorMap *map, const HalfOperand &o, const uint16_t *h, int box_rows) {
  PFN_cuTensorMapEncodeTiled_v12000 fn = get_encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t pitch = static_cast<cuuint64_t>(o.p.pitch) * 2;
  cuuint32_t estr[3] = {1, 1, 1};
  if (h == nullptr) return false;   // (the panels of this reading were not made)
  if (!o.cols) {
    cuuint64_t gdim[2] = {static_cast<cuuint64_t>(o.k), static_cast<cuuint64_t>(o.rows)};
    cuuint64_t gstride[1] = {pitch};
    cuuint32_t box[2] = {HG_BK, static_cast<cuuint32_t>(box_rows)};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<uint16_t *>(h), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  // 64 operand rows (128 bytes) x K x chunks of 64 rows: a box lands chunk after chunk, each chunk 64 K rows of 128 bytes
  cuuint64_t gdim[3] = {64, static_cast<cuuint64_t>(o.k), static_cast<cuuint64_t>((o.rows + 63) / 64)};
  cuuint64_t gstride[2] = {pitch, 128};
  cuuint32_t box[3] = {64, HG_BK, static_cast<cuuint32_t>(box_rows / 64)};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<uint16_t *>(h), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static inline long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }
static size_t scale_floats(long long R, long long C) {   // of the panels read through R rows
  return static_cast<size_t>(round_up(R, HP_BLOCK) / 2) * static_cast<size_t>((C + HP_BLOCK - 1) / HP_BLOCK);
}

size_t half_panel_floats(long long R, long long C, int readings) {
  size_t n = 64;   // alignment of the base
  if (readings & HALF_ROWS) n += static_cast<size_t>(R * round_up(C, 64)) + scale_floats(R, C);
  if (readings & HALF_COLS) n += static_cast<size_t>(R * round_up(C, 64)) + scale_floats(C, R);
  return n;
}

HalfPanels half_panels_at(float *mem, long long R, long long C, int readings) {
  HalfPanels p;
  p.R = R; p.C = C; p.pitch = round_up(C, 64);
  mem = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(mem) + 255) & ~static_cast<uintptr_t>(255));
  auto place = [&](HalfReading &to, long long rows, long long k) {   // (every part is a multiple of 64 floats or, an array of halves, of 32)
    to.h0 = reinterpret_cast<uint16_t *>(mem);
    to.h1 = to.h0 + R * p.pitch;
    to.scale = to.h1 + R * p.pitch;
    to.pitch = round_up(rows, HP_BLOCK);
    mem += R * p.pitch + static_cast<long long>(scale_floats(rows, k));
  };
  if (readings & HALF_ROWS) place(p.rows, R, C);
  if (readings & HALF_COLS) place(p.cols, C, R);
  return p;
}

HalfOperand half_rows(const HalfPanels &p) {
  HalfOperand o;
  o.p = p; o.cols = false; o.rows = p.R; o.k = p.C;
  return o;
}
HalfOperand half_cols(const HalfPanels &p) {
  HalfOperand o;
  o.p = p; o.cols = true; o.rows = p.C; o.k = p.R;
  return o;
}

int half_split(Context &ctx, const float *src, long long stride, const HalfPanels &p, const RowSegments *seg) {
  if (src == nullptr || (p.rows.h0 == nullptr && p.cols.h0 == nullptr) || p.R <= 0 || p.C <= 0) return MYEA_E_INVALID;
  SplitSource f;
  f.src = src;
  f.stride = stride;
  if (seg != nullptr) f.seg = *seg;
  f.vec = ((stride | f.seg.seg_off[0] | f.seg.seg_off[1] | f.seg.seg_off[2] | f.seg.seg_off[3]) & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  ctx.begin(TC_SPLIT);
  half_produce(ctx, f, p);
  ctx.end(TC_SPLIT);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

bool epilogue_takes_stats(const Context &ctx, const Epilogue &e, long long N) {
  if (ctx.gemm_engine != 0 || (N & 31) != 0 || e.ldc != N || e.seg_rows != 0 || !derivative_is_fused(e.deriv_af)) return false;
  if (((reinterpret_cast<uintptr_t>(e.col_stats) | reinterpret_cast<uintptr_t>(e.col_mean)) & 15) != 0) return false;
  const int v = epilogue_variant(e);
  return v == EPI_PLAIN_STATS || v == EPI_PRE_STATS || v == EPI_Y_STATS || v == EPI_BOTH_STATS;
}

// Workspace of split tiles: two partial-sum slots of one 256 x 256 tile per cluster and one arrival counter per (split
// tile, warp region).  Without it the kernel computes whole tiles only.
int gemm_splitk_reserve(Context &ctx) {
  if (ctx.sk_ws != nullptr) return MYEA_OK;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device) != cudaSuccess || sms < 2) return MYEA_E_CUDA;
  const int clusters = sms / 2;
  const size_t floats = static_cast<size_t>(clusters) * 2 * 16 * HG_REGION_FLOATS;
  if (cudaMalloc(&ctx.sk_ws, floats * sizeof(float)) != cudaSuccess) { ctx.sk_ws = nullptr; return MYEA_E_CUDA; }
  if (cudaMalloc(&ctx.sk_counters, static_cast<size_t>(clusters) * 16 * sizeof(unsigned int)) != cudaSuccess ||
      cudaMemset(ctx.sk_counters, 0, static_cast<size_t>(clusters) * 16 * sizeof(unsigned int)) != cudaSuccess) {
    cudaFree(ctx.sk_ws);
    ctx.sk_ws = nullptr;
    return MYEA_E_CUDA;
  }
  ctx.sk_clusters = clusters;
  return MYEA_OK;
}
void gemm_splitk_release(Context &ctx) {
  if (ctx.sk_ws != nullptr) cudaFree(ctx.sk_ws);
  if (ctx.sk_counters != nullptr) cudaFree(ctx.sk_counters);
  ctx.sk_ws = nullptr;
  ctx.sk_counters = nullptr;
  ctx.sk_clusters = 0;
}

// How `tiles` of `chunks` chunks of K are shared by `pairs` CTA pairs: whole ones in full waves, stream-K for the partial last wave.
struct WideSplit {
  int whole, run, clusters;   // tiles computed whole; chunks per cluster of the others (0: none); clusters of the launch
};
static WideSplit split_tiles(int tiles, int chunks, int pairs) {
  const int rem = tiles % pairs, units = rem * chunks;
  const WideSplit none = {tiles, 0, std::min(tiles, pairs)};
  if (rem == 0 || chunks < 2) return none;
  // at most 8 clusters share one tile: the cluster that arrives last adds up every other contributor's 256 KB of
  // partial sums, and past 8 that pass outweighs the shorter K walk (256 x 256 x 16384 with the splits of its operands 58 us, 94 with
  // 64 of them; 512 x 512 x 8192 50, 55 with 16)
  constexpr int max_split = 8;
  int run = std::max((units + pairs - 1) / pairs, (chunks + max_split - 1) / max_split);
  // A run that ends inside a tile makes a third contributor and a second set of partial sums (7 - 9 kcycles at the end of a
  // launch that walks a chunk in 3): where equal shares of a tile are hardly longer, every run is one share of one tile.
  // 32 tiles on 74 pairs, 16 chunks instead of 14: 512 x 4096 x 4096 with the splits of its operands 84.7 -> 78.9 us.  Two chunks more
  // pay at the shortest K as well: 25 tiles of 8 chunks, 4 instead of 3 37.1 -> 31.8; 26 of 16, 8 instead of 6 51.9 -> 46.5; 15 of 9, 3
  // instead of 2 35.9 -> 30.7.
  if (tiles == rem) {
    const int shares = std::min(pairs / rem, max_split), share = (chunks + shares - 1) / shares;
    if (share - run <= 2 && chunks % share == 0) run = share;
  }
  // splitting a tile costs about the time of two chunks (partial sums through L2, one counter round trip, the second
  // pass of the warp that arrives last): worth it when it takes at least three off the longest cluster
  if (chunks - run < 3) return none;
  return {tiles - rem, run, tiles > rem ? pairs : (units + run - 1) / run};
}

template <int BN, bool A_COLS, bool B_COLS>
static int launch_half(Context &ctx, const HalfOperand &A, const HalfOperand &B, const GemmDims &dims, const Epilogue &epi) {
  auto kernel = half_gemm_kernel<BN, A_COLS, B_COLS>;
  using S = HalfSmem<BN>;
  static PerDeviceOnce once;  // value: clusters of two CTAs that can be resident at once on the device
  const int device = ctx.device;
  const int G = once.get(device, [kernel, device] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL) != cudaSuccess) return 0;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 2) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(sms & ~1));
    cfg.blockDim = dim3(HG_THREADS);
    cfg.dynamicSmemBytes = S::TOTAL;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = sms / 2;
    }
    return n < sms / 2 ? n : sms / 2;
  });
  if (G <= 0) return MYEA_E_CUDA;
  CUtensorMap maps[4];
  if (!make_half_map(&maps[0], A, A.reading().h0, 128) || !make_half_map(&maps[1], A, A.reading().h1, 128) ||
      !make_half_map(&maps[2], B, B.reading().h0, BN / 2) || !make_half_map(&maps[3], B, B.reading().h1, BN / 2))
    return MYEA_E_CUDA;
  auto scales = [](const HalfOperand &o) {
    return ScaleView{o.reading().scale, o.reading().pitch, static_cast<int>((o.rows - 1) / HP_BLOCK)};
  };
  const int num_kb = (dims.K + HG_BK - 1) / HG_BK;
  const int num_chunks = (num_kb + HG_KC - 1) / HG_KC;
  WideWork work = {};
  work.tiles_m = (dims.M + 255) / 256;
  work.tiles_n = (dims.N + BN - 1) / BN;
  work.num_tiles = work.tiles_m * work.tiles_n;
  work.dp_tiles = work.num_tiles;
  int grid_clusters = std::min(work.num_tiles, G);
  // (gemm_bn 4 switches the split off; it needs the partial-sum workspace)
  if (ctx.gemm_bn != 4 && ctx.sk_ws != nullptr && ctx.sk_clusters >= G) {
    const WideSplit split = split_tiles(work.num_tiles, num_chunks, G);
    if (split.run > 0) {
      work.dp_tiles = split.whole;
      work.sk_units = (work.num_tiles - split.whole) * num_chunks;
      work.sk_chunks = split.run;
      work.ws = ctx.sk_ws;
      work.counters = ctx.sk_counters;
      grid_clusters = split.clusters;
    }
  }
  launch_dependent(ctx, kernel, dim3(static_cast<unsigned>(2 * grid_clusters)), dim3(HG_THREADS), S::TOTAL, maps[0], maps[1], maps[2], maps[3], scales(A), scales(B), dims,
                   work, epi, epilogue_variant(epi), ctx.d_error_flag);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

int half_gemm(Context &ctx, const HalfOperand &A, const HalfOperand &B, const Epilogue &epi) {
  const long long M = A.rows, N = B.rows, K = A.k;
  if (B.k != K || M <= 0 || N <= 0 || K <= 0) return MYEA_E_INVALID;
  for (const HalfOperand *o : {&A, &B})
    if (o->rows > (o->cols ? o->p.C : o->p.R) || K > (o->cols ? o->p.R : o->p.C) || o->reading().h0 == nullptr) return MYEA_E_INVALID;
  if (!derivative_is_fused(epi.deriv_af)) {
    if (epi.accumulate || epi.seg_rows != 0 || epi.stats_kind != 0 || epi.ldc != N || epi.ld_aux != N) return MYEA_E_UNSUPPORTED;
    Epilogue plain = epi;
    plain.deriv_af = 0;
    const int rc = half_gemm(ctx, A, B, plain);
    return rc != MYEA_OK ? rc : activation_backward(ctx, epi.C, epi.aux_pre, epi.aux_y, M, N, epi.deriv_af, epi.col_scale, epi.col_shift);
  }
  GemmDims dims{static_cast<int>(M), static_cast<int>(N), static_cast<int>(K)};
  ctx.begin(TC_GEMM);
  int rc;
  const int which = (A.cols ? 2 : 0) + (B.cols ? 1 : 0);
  if (N <= 128) {
    rc = which == 0 ? launch_half<128, false, false>(ctx, A, B, dims, epi) : which == 1 ? launch_half<128, false, true>(ctx, A, B, dims, epi)
       : which == 2 ? launch_half<128, true, false>(ctx, A, B, dims, epi) : launch_half<128, true, true>(ctx, A, B, dims, epi);
  } else {
    rc = which == 0 ? launch_half<256, false, false>(ctx, A, B, dims, epi) : which == 1 ? launch_half<256, false, true>(ctx, A, B, dims, epi)
       : which == 2 ? launch_half<256, true, false>(ctx, A, B, dims, epi) : launch_half<256, true, true>(ctx, A, B, dims, epi);
  }
  ctx.end(TC_GEMM);
  ctx.gemm_flops += 2.0 * dims.M * dims.N * static_cast<double>(dims.K);
  return rc;
}

size_t gemm_scratch_floats(long long M, long long N, long long K) {
  // whichever index of an operand is contiguous in memory
  return std::max(half_panel_floats(M, K, HALF_ROWS), half_panel_floats(K, M, HALF_COLS)) +
         std::max(half_panel_floats(N, K, HALF_ROWS), half_panel_floats(K, N, HALF_COLS));
}

int gemm_nt(Context &ctx, const Operand &A, const Operand &B, const Epilogue &epi, const GemmScratch &scratch) {
  if (A.k != B.k || A.rows <= 0 || B.rows <= 0 || A.k <= 0) return MYEA_E_INVALID;
  if (ctx.gemm_engine == 1) {  // the FP32 FMA engine
    GemmDims dims{static_cast<int>(A.rows), static_cast<int>(B.rows), static_cast<int>(A.k)};
    ctx.begin(TC_GEMM);
    dim3 grid(static_cast<unsigned>((dims.N + 63) / 64), static_cast<unsigned>((dims.M + 63) / 64));
    gemm_fp32_fma_kernel<<<grid, 256, 0, ctx.stream>>>(A, B, dims, epi);
    ctx.end(TC_GEMM);
    ctx.gemm_flops += 2.0 * dims.M * dims.N * static_cast<double>(dims.K);
    return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
  }
  if (epi.stats_kind == 0 && direct_gemm_suits(ctx, A.rows, B.rows, A.k)) {
    const DirectItem item{A, B, epi, nullptr};
    return direct_gemm(ctx, &item, 1);
  }
  auto need = [](const Operand &o) { return o.stride_k != 1 ? half_panel_floats(o.k, o.rows, HALF_COLS) : half_panel_floats(o.rows, o.k, HALF_ROWS); };
  if (scratch.base == nullptr || scratch.floats < need(A) + need(B)) return MYEA_E_INVALID;
  float *mem = scratch.base;
  HalfOperand ops[2];
  for (int i = 0; i < 2; ++i) {
    const Operand &o = i == 0 ? A : B;
    const bool cols = o.stride_k != 1;   // the operand's rows are contiguous: split as it lies, read through its columns
    const HalfPanels p = cols ? half_panels_at(mem, o.k, o.rows, HALF_COLS) : half_panels_at(mem, o.rows, o.k, HALF_ROWS);
    const int rc = half_split(ctx, o.ptr, cols ? o.stride_k : o.stride_r, p);
    if (rc != MYEA_OK) return rc;
    ops[i] = cols ? half_cols(p) : half_rows(p);
    mem += need(o);
  }
  return half_gemm(ctx, ops[0], ops[1], epi);
}

}  // namespace myea

// For tests: how `tiles` output tiles with `chunks` chunks of 128 of K are shared by `pairs` CTA pairs.  whole: tiles computed whole; run: chunks
// per pair of the others, 0 if there are none; clusters: pairs of the launch.
extern "C" int myea_b200_split_plan(int tiles, int chunks, int pairs, int *whole, int *run, int *clusters) {
  if (tiles <= 0 || chunks <= 0 || pairs <= 0 || whole == nullptr || run == nullptr || clusters == nullptr) return MYEA_E_INVALID;
  const myea::WideSplit s = myea::split_tiles(tiles, chunks, pairs);
  *whole = s.whole;
  *run = s.run;
  *clusters = s.clusters;
  return MYEA_OK;
}
