// All time steps of one LSTM layer and direction in ONE launch.
//
// The reference walks time strictly serially: per step the recurrent products of the four gates, the gate / cell /
// peephole arithmetic, then the next step (forward: Neural_Network__Recurrent_Forward_Pass__OpenMP.cpp:448-471 with the
// gates at :859-1040; BPTT: Neural_Network__Recurrent_Backward_Pass__OpenMP.cpp:440-862 with :1130-1604).  Launching a
// contraction and a cell kernel per step leaves the GPU waiting on launches: a step is 2 GFLOP.  Here one kernel stays
// resident for the whole walk:
//
//   grid      one cluster of SPLIT CTAs per 128 x BN tile of the step's product; the CTAs of a cluster share the tile and
//             split its K range (forward: BN = 128 gate columns, K = cells in 2 slices; backward: BN = 64 cells, K = 4 x
//             cells in 4 slices: 8-CTA clusters would halve the weight traffic per SM, but a B200 holds only 15 of the 16
//             a layer of 1024 cells needs), so that every SM streams a small share of the recurrent weights per step
//             (they do not fit shared memory; they stay in L2)
//   operands  half panels (half_panels.cuh): 4 bytes per element.  The gate rows of the weights are ordered (group of 16
//             cells, gate, cell): forward reads the tensor's rows, backward its columns, each with one power of two for all of
//             their K.  h is at most 1 in magnitude and has a fixed exponent; the gate errors have one exponent per batch row and
//             group of 16 cells - the 64 of K that one CTA produces and that one stage of a later step consumes
//   warp 0    TMA producer: waits until the operand panels of the previous step are complete (step barrier), then
//             loads its K slice of the step's operand (h of step s-1, or the gate errors of step s-1 of the walk) and
//             of the recurrent weights, 64 of K per stage
//   warp 1    one lane issues tcgen05.mma (h1*h0 + h0*h1 + h0*h0 per 16 of K) into a ring of accumulators in tensor memory
//   warps 4-11 take the partial sums out of tensor memory, backward times the power of two of their batch row, and exchange
//             them inside the cluster: every thread pushes the columns that other CTAs finish into those CTAs' shared
//             memory (st.async: the receiver's barrier counts the bytes, the sender waits for nothing) and keeps its own; the sums are added in slice order (bitwise
//             repeatable).  Each thread then finishes 8 cells of one batch row: gates, peepholes, cell state, zoneout keep
//             (forward) or the gate errors (backward).  The operand panels of the next step are stored before the step
//             barrier; the layer's arrays, which only later kernels read, after it.  What the cell needs from global
//             memory is fetched before the wait for the tensor cores.
//   step barrier: every CTA of a row of tiles counts itself in on a global counter when its results of step s are
//             written; producers poll it before they load step s + 1.  Every wait in the kernel is bounded (about a
//             second of SM clock): a wait that runs out sets the handle's error flag and an abort word that makes all
//             other waits give up, the CTAs wait (bounded as well) until every copy into their shared memory and every product
//             has landed, meet at their final barriers, free tensor memory and return.
// The launch needs all its CTAs resident at once (they wait for each other): lstm_persistent_plan checks the tile count
// against cudaOccupancyMaxActiveClusters and the layer falls back to one launch pair per step otherwise.
#include "half_panels.cuh"
#include "lstm.cuh"
#include "panel_math.cuh"
#include "tcgen05.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace myea {

// three warpgroups: warps 0-3 hold the two single-thread roles (warps 2-3 idle) and give most of their registers away
// (setmaxnreg); warps 4-11 exchange and run the cells with 232 registers each
constexpr int PS_THREADS = 384;
constexpr int PS_EPI_WARP0 = 4;
constexpr int PS_EPI_THREADS = 256;
constexpr int PS_BK = 64;                            // K per stage
constexpr int PS_A_BYTES = 128 * 128;                // 128 operand rows x 64 halves
// shapes of the two kernels: BN columns per tile, SPLIT K slices (= CTAs per cluster), SETS of columns per accumulator: with
// two, a0 * [b0 b1] is one instruction of twice the width (the two halves of the weights lie one behind the other in a stage),
// so that a0 is read from shared memory once for both.  Shared memory is what these narrow tiles wait for: 128 bytes per clock
// make 6 KB of operands per 128 x 64 x 16 product last 48 clocks where the product takes 32 (backward stage 1530 -> 1230
// clocks).  At 128 columns operands and product take 64 alike, and two sets leave a ring of two accumulators that the exchange
// warps do not empty in time (forward stage 1450 -> 1560 clocks).
template <int KIND> struct PsShape;
template <> struct PsShape<1> { static constexpr int BN = 128, SPLIT = 2, STAGES = 3, SETS = 1; };
template <> struct PsShape<2> { static constexpr int BN = 64, SPLIT = 4, STAGES = 4, SETS = 2; };
template <int KIND> struct PsSmem {
  static constexpr int BN = PsShape<KIND>::BN, STAGES = PsShape<KIND>::STAGES;
  static constexpr int B_BYTES = BN * 128;
  static constexpr int STAGE_BYTES = 2 * PS_A_BYTES + 2 * B_BYTES;     // A h0, A h1, B h0, B h1
  static constexpr int RECV_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int RECV_BYTES = (PsShape<KIND>::SPLIT - 1) * 128 * (BN / PsShape<KIND>::SPLIT) * 4;  // one slot per peer
  static constexpr int BAR_OFFSET = RECV_OFFSET + RECV_BYTES;
  static constexpr int SCALE_OFFSET = BAR_OFFSET + 512;                // powers of two of the columns this CTA finishes
  static constexpr int MAX_OFFSET = SCALE_OFFSET + BN / PsShape<KIND>::SPLIT * 4;   // backward: largest gate errors, [2 halves][128 rows]
  static constexpr int TOTAL = MAX_OFFSET + (KIND == 2 ? 2 * 128 * 4 : 0) + 1024;   // slack to align the base
  // Accumulators in tensor memory, used as a ring: the exchange warps read one while the tensor core fills the next ones.
  // Two sets: h0 * h0 and the cross products.
  static constexpr int TMEM_COLS = 512;
  static constexpr int ACC_COLS = PsShape<KIND>::SETS * BN;
  static constexpr int ACCS = TMEM_COLS / ACC_COLS;
  static_assert(STAGES <= 4, "a stage's done barrier is not reused before the stage is");
  static_assert(TOTAL <= 227 * 1024, "shared memory of one SM");
  static_assert(STAGE_BYTES % 1024 == 0 && B_BYTES % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
};

struct LstmSeq {
  int T = 0, B = 0, C = 0;
  int reverse = 0;              // the direction's time runs from T-1 down to 0
  int tiles_m = 0, tiles_n = 0;
  int split = 1;                // CTAs per cluster = K slices per tile
  int kb_per = 0, num_kb = 0;   // stages of K per slice / in all
  long long ldh = 0;            // pitch of the layer's output / error rows
  long long a_rows = 0;         // rows of one of the two operand-panel buffers (a multiple of 128)
  long long kpa = 0;            // pitch of the operand panels
  uint16_t *a0 = nullptr, *a1 = nullptr;      // [2][a_rows][kpa]: step s reads buffer (s-1)&1 and writes buffer s&1
  uint16_t *a_scale = nullptr;                // backward: [2][tiles_m][num_kb][128] powers of two of the gate errors' rows
  const float *w_scale = nullptr;             // powers of two of the weights: of the gate rows forward, of the cells backward
  const float *peep = nullptr;                // [3][C]
  const float *gates_in = nullptr;            // [T*B, 4C]
  float *act = nullptr, *cstate = nullptr, *cact = nullptr;
  float *values = nullptr;                    // layer outputs, this direction's columns, pitch ldh
  const uint8_t *zone_state = nullptr, *zone_output = nullptr;  // [T][C] or null
  float *deriv = nullptr;                     // error on the outputs, this direction's columns, pitch ldh
  float *dgates = nullptr, *dcstate = nullptr;
  unsigned int *sync = nullptr;               // [tiles_m] step counters, then one abort word
  long long wait_cycles = 1ll << 31;          // limit of the wait at a step barrier
  int stall_step = 0;                         // tests only: the step whose barrier is never reached (0: none)
  int *error_flag = nullptr;
};

// the arrays of walk step s as the cell arithmetic wants them
template <int KIND>
__device__ __forceinline__ LstmStep step_view(const LstmSeq &q, int s) {
  LstmStep p;
  const long long B = q.B, C = q.C, T = q.T;
  p.C = C; p.ldh = q.ldh; p.kp = q.kpa;
  if (s + 1 < q.T) {
    p.p_h0 = q.a0 + static_cast<long long>(s & 1) * q.a_rows * q.kpa;
    p.p_h1 = q.a1 + static_cast<long long>(s & 1) * q.a_rows * q.kpa;
  }
  if (KIND == 1) {
    const long long t = q.reverse ? T - 1 - s : s;
    p.gates_in = q.gates_in + t * B * 4 * C;
    p.act = q.act + t * B * 4 * C;
    p.cstate = q.cstate + t * B * C;
    p.cact = q.cact + t * B * C;
    p.h = q.values + t * B * q.ldh;
    p.zone_state = q.zone_state != nullptr ? q.zone_state + t * C : nullptr;
    p.zone_output = q.zone_output != nullptr ? q.zone_output + t * C : nullptr;
  } else {
    const long long t = q.reverse ? s : T - 1 - s;        // the walk goes against the direction
    const long long tp = q.reverse ? t + 1 : t - 1;       // the step before t
    p.dh = q.deriv + t * B * q.ldh;
    p.b_act = q.act + t * B * 4 * C;
    p.b_cact = q.cact + t * B * C;
    p.b_c_prev = (tp >= 0 && tp < T) ? q.cstate + tp * B * C : nullptr;
    p.dgates = q.dgates + t * B * 4 * C;
    p.dcstate = q.dcstate + t * B * C;
  }
  return p;
}

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed_gpu(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int *p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait for a step counter; gives up when any CTA has raised the abort word or after about a second.  The counter is
// polled alone (the abort word every 64 looks: a second round trip per look delayed every step by half of it).
__device__ __forceinline__ bool wait_step_counter(const unsigned int *counter, unsigned int target, const unsigned int *abort_word, volatile int *abort_flag,
                                                  long long limit) {
  if (*abort_flag) return false;
  const long long t0 = clock64();
  for (int look = 0; ld_relaxed_gpu(counter) < target; ++look) {
    if ((look & 63) == 63 && (ld_relaxed_gpu(abort_word) != 0u || clock64() - t0 > limit)) {
      *abort_flag = 1;
      return false;
    }
  }
  return ld_acquire_gpu(counter) >= target;   // (orders what follows after the other CTAs' stores)
}

template <int KIND>
__global__ void __launch_bounds__(PS_THREADS, 1)
lstm_persistent_kernel(const __grid_constant__ CUtensorMap tm_a0, const __grid_constant__ CUtensorMap tm_a1,
                       const __grid_constant__ CUtensorMap tm_b0, const __grid_constant__ CUtensorMap tm_b1, const LstmSeq q) {
  using SM = PsSmem<KIND>;
  constexpr int STAGES = SM::STAGES, BN = SM::BN, S = PsShape<KIND>::SPLIT, ACCS = SM::ACCS, DONE = 4, SETS = PsShape<KIND>::SETS;
  constexpr int W = BN / S;   // columns of the tile this CTA finishes: 16 cells (x 4 gates forward)
  extern __shared__ uint8_t smem_raw[];
  // the dynamic shared-memory window starts at the same offset in every CTA of the cluster, so the aligned offsets
  // (and with them the addresses peers compute for each other's buffers and barriers) match as well
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float *recv = reinterpret_cast<float *>(smem + SM::RECV_OFFSET);  // [S - 1 peers][128 rows][W]: partial sums pushed by the peers
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(smem + SM::BAR_OFFSET);
  uint64_t *done_bar = full_bar + STAGES;    // [DONE] the products of a stage are done: its accumulator is complete, the stage free
  uint64_t *acc_empty = done_bar + DONE;     // [ACCS] the 8 exchange warps have read the accumulator
  uint64_t *red_ready = acc_empty + ACCS;    // the peers' partial sums for this CTA have landed
  uint64_t *step_go = red_ready + 1;         // the producer has passed the step barrier
  uint64_t *drained = step_go + 1;           // a wait has given up: the products issued so far are done
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(drained + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);
  uint32_t *left_early = tmem_holder + 2;    // a wait of this cluster has given up
  uint32_t *pushed_s = tmem_holder + 3, *armed_s = tmem_holder + 4;   // threads' pushes, and steps whose pushes were expected, in all
  float *scale_s = reinterpret_cast<float *>(smem + SM::SCALE_OFFSET);
  float *max_s = reinterpret_cast<float *>(smem + SM::MAX_OFFSET);
  float *peep_s = reinterpret_cast<float *>(smem + SM::BAR_OFFSET + 320);  // [3][16] peepholes of this CTA's cells

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int cluster_id = static_cast<int>(blockIdx.x) / S;
  const int tile_m = cluster_id / q.tiles_n, tile_n = cluster_id - tile_m * q.tiles_n;
  const int m0 = tile_m * 128, n0 = tile_n * BN;
  const int kb0 = min(static_cast<int>(rank) * q.kb_per, q.num_kb), kb1 = min(kb0 + q.kb_per, q.num_kb);
  const int my_kb = kb1 - kb0;
  unsigned int *counter = q.sync + tile_m;
  unsigned int *abort_word = q.sync + q.tiles_m;
  const unsigned int per_step = static_cast<unsigned int>(q.tiles_n * S);  // CTAs that complete a row of tiles

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) ptx::mbar_init(&full_bar[s], 1);
    for (int s = 0; s < DONE; ++s) ptx::mbar_init(&done_bar[s], 1);
    for (int a = 0; a < ACCS; ++a) ptx::mbar_init(&acc_empty[a], 8);
    ptx::mbar_init(red_ready, 1);
    ptx::mbar_init(step_go, 1);
    ptx::mbar_init(drained, 1);
    *abort_flag = 0;
    *left_early = *pushed_s = *armed_s = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_holder, SM::TMEM_COLS);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // every CTA's barriers exist before anyone signals across the cluster
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  uint32_t issued = 0;  // producer: K blocks staged so far (for the final drain)
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    ptx::reg_release<40>();
    if (lane == 0) {
      bool ok = true;
      auto wait_free = [&](uint32_t u) {   // the stage's last products are done
        const uint32_t v = u - static_cast<uint32_t>(STAGES);
        return u < static_cast<uint32_t>(STAGES) || ptx::mbar_wait_or_abort(&done_bar[v % DONE], (v / DONE) & 1u, abort_flag);
      };
      auto load_a = [&](uint32_t u, int kb, int a_row) {
        uint8_t *dst = smem + (u % STAGES) * SM::STAGE_BYTES;
        ptx::tma_load_2d(dst, &tm_a0, &full_bar[u % STAGES], kb * PS_BK, a_row);
        ptx::tma_load_2d(dst + PS_A_BYTES, &tm_a1, &full_bar[u % STAGES], kb * PS_BK, a_row);
      };
      auto load_b = [&](uint32_t u, int kb) {
        uint8_t *dst = smem + (u % STAGES) * SM::STAGE_BYTES + 2 * PS_A_BYTES;
        if constexpr (KIND == 1) {
          ptx::tma_load_2d(dst, &tm_b0, &full_bar[u % STAGES], kb * PS_BK, n0);
          ptx::tma_load_2d(dst + SM::B_BYTES, &tm_b1, &full_bar[u % STAGES], kb * PS_BK, n0);
        } else {
          ptx::tma_load_3d(dst, &tm_b0, &full_bar[u % STAGES], 0, kb * PS_BK, n0 >> 6);
          ptx::tma_load_3d(dst + SM::B_BYTES, &tm_b1, &full_bar[u % STAGES], 0, kb * PS_BK, n0 >> 6);
        }
      };
      for (int s = 1; s < q.T && ok; ++s) {
        // the weights of the step's first stages do not depend on the step before: they are on their way before the barrier
        const int ahead = min(STAGES, my_kb);
        int loaded = 0;
        for (; loaded < ahead; ++loaded) {
          const uint32_t u = issued + static_cast<uint32_t>(loaded);
          if (!wait_free(u)) { ok = false; break; }
          ptx::mbar_arrive_expect_tx(&full_bar[u % STAGES], SM::STAGE_BYTES);
          load_b(u, kb0 + loaded);
        }
        if (ok) ok = wait_step_counter(counter, per_step * static_cast<unsigned int>(s) + (s == q.stall_step ? 1u : 0u), abort_word, abort_flag, q.wait_cycles);
        ptx::fence_proxy_async_global();  // the other CTAs wrote them with ordinary stores; TMA reads through the async proxy
        const int a_row = ((s - 1) & 1) * static_cast<int>(q.a_rows) + m0;
        // (after a wait that gave up as well, whatever lies there: the barriers of the weights on their way complete, so that the
        // exit below can wait for them)
        for (int i = 0; i < loaded; ++i) load_a(issued + static_cast<uint32_t>(i), kb0 + i, a_row);
        issued += static_cast<uint32_t>(loaded);
        if (!ok) break;
        // only now may the other warps store the arrays of the step before: their stores would keep these copies waiting
        ptx::mbar_arrive_local(step_go);
        for (int kb = kb0 + ahead; kb < kb1; ++kb, ++issued) {
          if (!wait_free(issued)) { ok = false; break; }
          ptx::mbar_arrive_expect_tx(&full_bar[issued % STAGES], SM::STAGE_BYTES);
          load_a(issued, kb, a_row);
          load_b(issued, kb);
        }
      }
      if (!ok) {
        atomicCAS(q.error_flag, 0, 401);
        atomicExch(abort_word, 1u);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    ptx::reg_release<40>();
    if (lane == 0) {
      bool ok = true;
      constexpr uint32_t idesc = make_idesc_f16(128, BN, false, KIND == 2), idesc2 = make_idesc_f16(128, SETS * BN, false, KIND == 2);
      constexpr uint64_t b_step = KIND == 2 ? 128 : 2;
      uint32_t it = 0;  // stages consumed = accumulators filled
      // the barriers of the next stage are asked before this one's instructions are issued (see half_gemm.cu)
      bool full_ok = false, acc_ok = false;
      for (int s = 1; s < q.T && ok; ++s) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t a = it % ACCS, st = it % STAGES;
          if (it >= ACCS) {
            if (!acc_ok && !ptx::mbar_wait_or_abort(&acc_empty[a], (it / ACCS - 1u) & 1u, abort_flag)) { ok = false; break; }
          }
          if (!full_ok && !ptx::mbar_wait_or_abort(&full_bar[st], (it / STAGES) & 1u, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after();
          full_ok = ptx::mbar_test(&full_bar[(it + 1) % STAGES], ((it + 1) / STAGES) & 1u);
          acc_ok = it + 1 >= ACCS && ptx::mbar_test(&acc_empty[(it + 1) % ACCS], ((it + 1) / ACCS - 1u) & 1u);
          const uint32_t t_acc = tmem_base + a * static_cast<uint32_t>(SM::ACC_COLS);
          const uint32_t base = ptx::smem_u32(smem + st * SM::STAGE_BYTES), base_b = base + 2 * PS_A_BYTES;
          const uint64_t a0 = make_smem_desc(base), a1 = make_smem_desc(base + PS_A_BYTES);
          const uint64_t b0 = KIND == 2 ? make_smem_desc_mn(base_b, 8192, false) : make_smem_desc(base_b);
#pragma unroll
          for (int k = 0; k < PS_BK / 16; ++k) {
            const uint64_t ka = static_cast<uint64_t>(k) * 2, kbo = static_cast<uint64_t>(k) * b_step;
            if constexpr (SETS == 2) {
              ptx::mma_bf16(t_acc, a0 + ka, b0 + kbo, idesc2, k > 0 ? 1u : 0u);   // a0 * b0 and a0 * b1
              ptx::mma_bf16(t_acc + BN, a1 + ka, b0 + kbo, idesc, 1u);            // a1 * b0 onto a0 * b1
            } else {
              const uint64_t b1 = make_smem_desc(base_b + SM::B_BYTES);
              ptx::mma_bf16(t_acc, a1 + ka, b0 + kbo, idesc, k > 0 ? 1u : 0u);
              ptx::mma_bf16(t_acc, a0 + ka, b1 + kbo, idesc, 1u);
              ptx::mma_bf16(t_acc, a0 + ka, b0 + kbo, idesc, 1u);
            }
          }
          // one commit per stage: the accumulator is complete and the stage free (a second one right behind it stalls the
          // issuer for 600 cycles)
          ptx::tc_commit(&done_bar[it % DONE]);
        }
      }
      if (!ok) {
        atomicCAS(q.error_flag, 0, 402);
        atomicExch(abort_word, 1u);
      }
    }
  } else if (warp >= PS_EPI_WARP0) {
    // ---------------- exchange + cell: 8 warps; tensor-memory lane quarter = warp % 4, half of the CTA's cells = (warp - 4) / 4 ----------------
    ptx::reg_acquire<232>();
    constexpr int HW = W / 2;   // this thread's columns of its CTA's share: 8 cells (x 4 gates forward)
    constexpr int CW = W / 4;   // 16-byte chunks per row of a receive slot
    static_assert((KIND == 1 ? BN / 4 : BN) / S == 16 && (HW == 32 || HW == 8), "16 cells per CTA, 8 per thread");
    const int qd = warp & 3, half = (warp - PS_EPI_WARP0) >> 2;
    const int row = qd * 32 + lane;
    const int swz = CW == 16 ? (row & 15) : ((row >> 1) & 3);  // chunk swizzle of the receive slots (bank conflicts)
    const long long b = static_cast<long long>(m0) + row;
    // a tile holds 32 cells x 4 gates (forward) or 64 cells (backward); this CTA finishes 16 of them, this thread 8
    const long long cta_cell0 = static_cast<long long>(tile_n) * (KIND == 1 ? BN / 4 : BN) + static_cast<long long>(rank) * 16;
    const long long cell0 = cta_cell0 + half * 8;
    const bool active = b < q.B && cell0 < q.C;
    const uint32_t recv_addr = ptx::smem_u32(recv);
    {  // the peepholes of this CTA's cells stay in shared memory for the whole walk
      const int i = static_cast<int>(threadIdx.x) - PS_EPI_WARP0 * 32;
      if (i < 48) {
        const long long cell = cta_cell0 + (i & 15);
        peep_s[i] = cell < q.C ? q.peep[static_cast<long long>(i >> 4) * q.C + cell] : 0.f;
      }
      // so do the powers of two of the columns it finishes (forward with the fixed one of h)
      const long long col = static_cast<long long>(n0) + static_cast<long long>(rank) * W + i;
      if (i < W) scale_s[i] = KIND == 1 ? (cta_cell0 < q.C ? q.w_scale[col] * pow2(LSTM_H_EXPONENT) : 0.f) : (col < q.C ? q.w_scale[col] : 0.f);
      ptx::named_barrier_sync(1, PS_EPI_THREADS);
    }
    using In = typename std::conditional<KIND == 1, LstmForwardIn, LstmBackwardIn>::type;
    using Out = typename std::conditional<KIND == 1, LstmForwardOut, LstmBackwardOut>::type;
    Out out;               // results of the step before; its arrays are written once the step barrier has been passed
    float fn[8];           // backward: the forget gates of the step of the walk before
#pragma unroll
    for (int i = 0; i < 8; ++i) fn[i] = 0.f;
    bool pending = false;
    uint32_t n = 0;        // accumulators read so far
    uint32_t pushed = 0, armed = 0;   // steps whose partial sums this thread has pushed / expects from the peers
    constexpr int ARRAYS = KIND == 1 ? LSTM_FORWARD_ARRAYS : LSTM_BACKWARD_ARRAYS;
    auto store_arrays = [&](int step, int first, int last) {
      const LstmStep pp = step_view<KIND>(q, step);
#pragma unroll
      for (int k = 0; k < ARRAYS; ++k) {
        if (k < first || k >= last) continue;
        if constexpr (KIND == 1) lstm_forward_store_array8(pp, out, b, cell0, k);
        else lstm_backward_store_array8(pp, out, b, cell0, k);
      }
    };
    // backward: power of two of this thread's row in accumulator c; asked for one accumulator ahead
    auto row_scale = [&](int step, int c) {
      const uint16_t *at = q.a_scale + ((static_cast<long long>((step - 1) & 1) * q.tiles_m + tile_m) * q.num_kb + kb0 + c) * 128 + row;
      return (static_cast<uint32_t>(__ldcg(at)) << 16) + (14u << 23);
    };
    for (int s = 0; s < q.T; ++s) {
      bool ok = true;
      const LstmStep p = step_view<KIND>(q, s);
      uint32_t next_scale = 0;
      In in;
      if (active) {
        // what the cell needs from global memory goes out before any wait; what this thread computed itself in the step
        // before (and has not written yet) comes from its registers
        if constexpr (KIND == 1) {
          lstm_forward_load8(p, in, b, cell0);
#pragma unroll
          for (int i = 0; i < 8; ++i) { in.cp[i] = s > 0 ? out.cs[i] : 0.f; in.hp[i] = s > 0 ? out.h[i] : 0.f; }
        } else {
          lstm_backward_load8(p, in, b, cell0);
#pragma unroll
          for (int i = 0; i < 8; ++i) { in.dni[i] = s > 0 ? out.di[i] : 0.f; in.dnf[i] = s > 0 ? out.df[i] : 0.f; in.dcn[i] = s > 0 ? out.dc[i] : 0.f; in.fn[i] = fn[i]; fn[i] = in.fg[i]; }
        }
      }
      if (pending) {
        // the arrays of step s - 1 (read by later kernels only) leave from here on, two per accumulator beside this step's
        // operand stream: all at once, the 128 CTAs' stores kept its first copies waiting (4 of a forward step's 30 kcycles), and
        // stored while the step barrier is in flight they slowed the barrier down
        if (!ptx::mbar_wait_or_abort(step_go, static_cast<uint32_t>(s - 1) & 1u, abort_flag)) ok = false;
        if (KIND == 2 && ok && my_kb > 0) next_scale = row_scale(s, 0);
      }
      float rec[HW];
#pragma unroll
      for (int i = 0; i < HW; ++i) rec[i] = 0.f;
      if (s > 0) {
        // Partial sums of this CTA's K slice: for every CTA d of the cluster the columns of d's cells that belong to this
        // thread's (row, half), added up over the accumulators as the tensor core completes them (part[S - 1] is this
        // CTA's own share, the others go to the peers in the order rank + 1, rank + 2, ...).  Forward: column g * 16 + cell
        // of a CTA's 64, kept as [gate][8 cells].
        float part[S][HW];
#pragma unroll
        for (int dd = 0; dd < S; ++dd)
#pragma unroll
          for (int j = 0; j < HW; ++j) part[dd][j] = 0.f;
        for (int c = 0; c < my_kb; ++c, ++n) {
          const uint32_t a = n % ACCS;
          const float sa = __uint_as_float(next_scale);
          if (KIND == 2 && c + 1 < my_kb) next_scale = row_scale(s, c + 1);
          if (!ptx::mbar_wait_or_abort(&done_bar[n % DONE], (n / DONE) & 1u, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after();
          const uint32_t tq = tmem_base + (static_cast<uint32_t>(qd * 32) << 16) + a * static_cast<uint32_t>(SM::ACC_COLS);
#pragma unroll
          for (int dd = 1; dd <= S; ++dd) {
            const int d = (static_cast<int>(rank) + dd) % S;
            constexpr int BATCH = HW / 8;   // 8-column groups per round trip
#pragma unroll
            for (int k0 = 0; k0 < HW / 8; k0 += BATCH) {
              uint32_t r[BATCH][8], x[BATCH][8];
#pragma unroll
              for (int k = 0; k < BATCH; ++k) {
                const uint32_t col = tq + static_cast<uint32_t>(d * W + (k0 + k) * 16 + half * 8);
                ptx::tmem_ld_32x8(col, r[k]);
                if constexpr (SETS == 2) ptx::tmem_ld_32x8(col + BN, x[k]);
              }
              ptx::tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < BATCH * 8; ++j) {
                float v = __uint_as_float(r[j / 8][j % 8]);
                if constexpr (SETS == 2) v += __uint_as_float(x[j / 8][j % 8]);
                float &t = part[dd - 1][k0 * 8 + j];
                t = KIND == 2 ? fmaf(v, sa, t) : t + v;
              }
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_local(&acc_empty[a]);
          if (active && 2 * c < ARRAYS) store_arrays(s - 1, 2 * c, 2 * c + 2);
        }
        if (ok && active && 2 * my_kb < ARRAYS) store_arrays(s - 1, 2 * my_kb, ARRAYS);
        pending = false;
        if (ok) {
          // the peers' shares are pushed into their receive slots, this CTA's own share stays in registers
#pragma unroll
          for (int dd = 1; dd < S; ++dd) {
            const int d = (static_cast<int>(rank) + dd) % S;
            const int slot = static_cast<int>(rank) < d ? static_cast<int>(rank) : static_cast<int>(rank) - 1;
            const uint32_t dst = ptx::map_to_cta(recv_addr + static_cast<uint32_t>((slot * 128 + row) * W * 4), static_cast<uint32_t>(d));
            const uint32_t bar = ptx::map_to_cta(ptx::smem_u32(red_ready), static_cast<uint32_t>(d));
#pragma unroll
            for (int i = 0; i < HW / 4; ++i)
              ptx::st_async_f4(dst + (static_cast<uint32_t>((half * (HW / 4) + i) ^ swz) << 4),
                               make_float4(part[dd - 1][4 * i], part[dd - 1][4 * i + 1], part[dd - 1][4 * i + 2], part[dd - 1][4 * i + 3]), bar);
          }
          ++pushed;
          if (warp == PS_EPI_WARP0 && lane == 0) {
            ptx::mbar_arrive_expect_tx(red_ready, static_cast<uint32_t>(SM::RECV_BYTES));
            ++armed;
          }
          if (!ptx::mbar_wait_cluster_or_abort(red_ready, static_cast<uint32_t>(s - 1) & 1u, abort_flag)) ok = false;
        }
        if (ok) {
          // the sums over the K slices, added in slice order whichever CTA adds them (bitwise repeatable)
#pragma unroll
          for (int j = 0; j < S; ++j) {
            if (j == static_cast<int>(rank)) {
#pragma unroll
              for (int i = 0; i < HW; ++i) rec[i] += part[S - 1][i];
            } else {
              const int slot = j < static_cast<int>(rank) ? j : j - 1;
              const float *src = recv + (slot * 128 + row) * W;
              float4 v[HW / 4];
#pragma unroll
              for (int i = 0; i < HW / 4; ++i) v[i] = *reinterpret_cast<const float4 *>(src + (((half * (HW / 4) + i) ^ swz) << 2));
#pragma unroll
              for (int i = 0; i < HW / 4; ++i) { rec[4 * i] += v[i].x; rec[4 * i + 1] += v[i].y; rec[4 * i + 2] += v[i].z; rec[4 * i + 3] += v[i].w; }
            }
          }
#pragma unroll
          for (int i = 0; i < HW; ++i) rec[i] *= scale_s[(i >> 3) * 16 + half * 8 + (i & 7)];
        }
      }
      float m = 0.f;   // backward: this thread's largest gate error
      if (ok) {
        if (active) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { in.pi[i] = peep_s[half * 8 + i]; in.pf[i] = peep_s[16 + half * 8 + i]; in.po[i] = peep_s[32 + half * 8 + i]; }
        }
        // the cell; only what the NEXT step's contraction reads (the operand panels) leaves before the step barrier
        if constexpr (KIND == 1) {
          if (active) {
            lstm_forward_compute8(in, rec, s == 0, out);
            if (p.p_h0 != nullptr) lstm_store_h_panels8(p, out.h, b, cell0);
          }
        } else if (active) {
          lstm_backward_compute8(in, rec, p.b_c_prev != nullptr, out);
#pragma unroll
          for (int i = 0; i < 8; ++i) m = fmaxf(fmaxf(m, fmaxf(finite_abs(out.dz[i]), finite_abs(out.di[i]))), fmaxf(finite_abs(out.df[i]), finite_abs(out.d_o[i])));
        }
        pending = true;
      }
      if constexpr (KIND == 2) {
        if (p.p_h0 != nullptr) {
          // one exponent per row for this CTA's 16 cells x 4 gates (a warp that gave up takes part: the barrier is for all)
          max_s[half * 128 + row] = m;
          ptx::named_barrier_sync(1, PS_EPI_THREADS);
          const int e = half_exponent(fmaxf(m, max_s[(half ^ 1) * 128 + row]));
          const int group = static_cast<int>(cta_cell0 >> 4);
          if (half == 0 && group < q.num_kb)
            q.a_scale[((static_cast<long long>(s & 1) * q.tiles_m + tile_m) * q.num_kb + group) * 128 + row] = half_scale_bits(e);
          if (active && ok) lstm_store_gate_panels8(p, out, pow2(-e), b, static_cast<long long>(group) * 64 + half * 8);
        }
      }
      // this thread's panel stores come before the TMA copies that the step barrier lets loose (generic -> async proxy)
      ptx::fence_proxy_async_global();
      if (!ok && lane == 0) {
        atomicCAS(q.error_flag, 0, 403);
        atomicExch(abort_word, 1u);
      }
      // the 8 warps stay in step and leave together: the barrier returns the OR of what each thread saw of the CTA's
      // abort flag (a warp that gave up has set it before it gets here), the same answer in every thread
      if (ptx::named_barrier_or(1, PS_EPI_THREADS, *abort_flag != 0)) { pending = false; break; }
      // the barrier above ordered every thread's panel stores before this thread; its release makes them visible to
      // the GPU together with the count
      if (warp == PS_EPI_WARP0 && lane == 0) red_release_gpu_add(counter, 1u);
    }
    if (pending && active) store_arrays(q.T - 1, 0, ARRAYS);
    atomicAdd(pushed_s, pushed);
    if (warp == PS_EPI_WARP0 && lane == 0) *armed_s = armed;
  } else {
    ptx::reg_release<40>();  // warps 2-3: no role, but the whole warpgroup has to give its registers back
  }

  // the producer makes sure none of its copies is still in flight before the CTA's shared memory goes away
  if (warp == 0 && lane == 0) {
    const uint32_t first = issued > static_cast<uint32_t>(STAGES) ? issued - STAGES : 0u;
    for (uint32_t i = first; i < issued; ++i) {
      if (!ptx::mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1u)) break;
    }
  }
  // peers may still be pushing into this CTA's receive slots or signalling its barriers: the cluster stays together until
  // everybody is here
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0) {
    for (int d = 0; d < S; ++d) ptx::st_cluster_u32(ptx::map_to_cta(ptx::smem_u32(left_early), static_cast<uint32_t>(d)), 1u);
  }
  ptx::cluster_sync_all();
  // A wait of the cluster has given up (every CTA of it sees that here): products may still be reading shared memory, and partial
  // sums whose step nobody finished may be on their way into the receive slots.  The first have a barrier of their own.  The
  // second are counted by red_ready: it is told which bytes will never come, or to expect those that nobody had asked for, and
  // then completes when the last one has landed.  A peer is at most one step ahead (it has passed the step barrier of the step
  // before, where this CTA counted itself in with that step's sums complete), so one phase is all that can be open.
  if (*reinterpret_cast<volatile uint32_t *>(left_early) != 0u) {
    if (warp == 1 && lane == 0) {
      ptx::tc_commit(drained);
      ptx::mbar_wait(drained, 0);
    }
    if (threadIdx.x == PS_EPI_WARP0 * 32) {
      uint32_t threads = 0;
      for (int d = 0; d < S; ++d)
        if (d != static_cast<int>(rank)) threads += ptx::ld_cluster_u32(ptx::map_to_cta(ptx::smem_u32(pushed_s), static_cast<uint32_t>(d)));
      const uint32_t sent = threads * (W / 2 * 4), expected = *armed_s * static_cast<uint32_t>(SM::RECV_BYTES);
      uint32_t phases = *armed_s;
      if (sent < expected) ptx::mbar_complete_tx(red_ready, expected - sent);
      if (sent > expected) {
        ptx::mbar_arrive_expect_tx(red_ready, sent - expected);
        ++phases;
      }
      if (phases > 0) ptx::mbar_wait(red_ready, (phases - 1u) & 1u);
    }
    __syncthreads();
    ptx::cluster_sync_all();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, SM::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
struct LstmPersistent {
  bool ready = false;
  int tiles_m = 0;
  long long a_rows = 0;
  unsigned int *sync = nullptr;  // [tiles_m + 1]
  int stall_step = 0;            // see LstmSeq
  long long wait_cycles = 1ll << 31;
};

template <int KIND>
static int resident_clusters(int device) {
  constexpr int split = PsShape<KIND>::SPLIT;
  constexpr int PS_SMEM_TOTAL = PsSmem<KIND>::TOTAL;
  // clusters of `split` CTAs that fit the device at once; configured once per device (the shared-memory opt-in is a
  // per-device attribute of the kernel)
  static std::mutex mutex;
  static int cached[64] = {};
  if (device < 0 || device >= 64) return 0;
  std::lock_guard<std::mutex> lock(mutex);
  if (cached[device] != 0) return cached[device];
  auto kernel = lstm_persistent_kernel<KIND>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_SMEM_TOTAL) != cudaSuccess) { cudaGetLastError(); return 0; }
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sms / split * split));
  cfg.blockDim = dim3(PS_THREADS);
  cfg.dynamicSmemBytes = PS_SMEM_TOTAL;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
  cached[device] = n > 0 ? n : -1;
  return cached[device];
}

int lstm_persistent_plan(myea_b200_net *net, LayerPlan &L) {
  LstmPlan *P = L.lstm;
  P->persist = nullptr;
  if (P->C % 8 != 0 || net->ctx.gemm_engine != 0 || net->T < 2) return MYEA_OK;
  const long long B = net->B, C = P->C;
  const int tiles_m = static_cast<int>((B + 127) / 128);
  const long long fwd_clusters = tiles_m * ((P->G + PsShape<1>::BN - 1) / PsShape<1>::BN), bwd_clusters = tiles_m * ((C + PsShape<2>::BN - 1) / PsShape<2>::BN);
  const int fit_f = resident_clusters<1>(net->ctx.device), fit_b = resident_clusters<2>(net->ctx.device);
  if (fwd_clusters > fit_f || bwd_clusters > fit_b) return MYEA_OK;  // the CTAs of a launch wait for each other: all of them have to fit
  LstmPersistent *ps = new LstmPersistent();
  ps->tiles_m = tiles_m;
  ps->a_rows = static_cast<long long>(tiles_m) * 128;
  void *q = nullptr;
  if (cudaMalloc(&q, (tiles_m + 1) * sizeof(unsigned int)) != cudaSuccess) { delete ps; net->ctx.error = "cudaMalloc failed (LSTM step counters)"; return MYEA_E_CUDA; }
  net->allocations.push_back(q);
  ps->sync = static_cast<unsigned int *>(q);
  ps->ready = true;
  P->persist = ps;
  return MYEA_OK;
}

void lstm_persistent_destroy(LstmPlan *P) {
  if (P != nullptr) { delete P->persist; P->persist = nullptr; }
}

bool lstm_persistent_ready(const LstmPlan *P) { return P != nullptr && P->persist != nullptr && P->persist->ready; }

template <int KIND>
static int launch(myea_b200_net *net, LstmSeq &q, long long K, const HalfPanels &w) {
  Context &ctx = net->ctx;
  // operand panels: both ping-pong buffers in one map (row coordinate = buffer * a_rows + tile row)
  HalfOperand a;
  a.p.R = 2 * q.a_rows; a.p.C = K; a.p.pitch = q.kpa;
  a.rows = a.p.R; a.k = K;
  const HalfOperand b = KIND == 1 ? half_rows(w) : half_cols(w);
  CUtensorMap maps[4];
  if (!make_half_map(&maps[0], a, q.a0, 128) || !make_half_map(&maps[1], a, q.a1, 128) || !make_half_map(&maps[2], b, b.reading().h0, PsShape<KIND>::BN) ||
      !make_half_map(&maps[3], b, b.reading().h1, PsShape<KIND>::BN))
    return MYEA_E_CUDA;
  if (cudaMemsetAsync(q.sync, 0, (q.tiles_m + 1) * sizeof(unsigned int), ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(q.tiles_m * q.tiles_n * q.split));
  cfg.blockDim = dim3(PS_THREADS);
  cfg.dynamicSmemBytes = PsSmem<KIND>::TOTAL;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(q.split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ctx.begin(TC_GEMM);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, lstm_persistent_kernel<KIND>, maps[0], maps[1], maps[2], maps[3], q);
  ctx.end(TC_GEMM);
  ctx.gemm_flops += 2.0 * q.B * 4.0 * q.C * q.C * (q.T - 1);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

static void common_args(myea_b200_net *net, LayerPlan &L, int dir, LstmSeq &q) {
  LstmPlan *P = L.lstm;
  q.T = static_cast<int>(net->T); q.B = static_cast<int>(net->B); q.C = static_cast<int>(P->C);
  q.reverse = dir;
  q.tiles_m = P->persist->tiles_m;
  q.ldh = L.n_out;
  q.a_rows = P->persist->a_rows;
  q.peep = P->peep_compact + static_cast<size_t>(dir) * 3 * P->C;
  q.sync = P->persist->sync;
  q.stall_step = P->persist->stall_step;
  q.wait_cycles = P->persist->wait_cycles;
  q.error_flag = net->ctx.d_error_flag;
}

int lstm_persistent_forward(myea_b200_net *net, LayerPlan &L, int dir, bool zoneout) {
  LstmPlan *P = L.lstm;
  if (!lstm_persistent_ready(P)) return MYEA_E_UNSUPPORTED;
  const LstmDir &D = P->d[dir];
  LstmSeq q;
  common_args(net, L, dir, q);
  q.tiles_n = static_cast<int>((P->G + PsShape<1>::BN - 1) / PsShape<1>::BN);
  q.split = PsShape<1>::SPLIT;
  q.num_kb = static_cast<int>((P->C + PS_BK - 1) / PS_BK);
  q.kb_per = (q.num_kb + q.split - 1) / q.split;
  q.kpa = P->h_pan.pitch;
  q.a0 = P->h_pan.rows.h0; q.a1 = P->h_pan.rows.h1;
  q.w_scale = P->w_rec_scale[dir];
  q.gates_in = D.gates_in; q.act = D.act; q.cstate = D.cstate; q.cact = D.cact;
  q.values = L.values + dir * P->C;
  q.zone_state = zoneout ? D.zone_state : nullptr;
  q.zone_output = zoneout ? D.zone_output : nullptr;
  return launch<1>(net, q, P->C, P->w_rec[dir]);
}

int lstm_persistent_backward(myea_b200_net *net, LayerPlan &L, int dir) {
  LstmPlan *P = L.lstm;
  if (!lstm_persistent_ready(P)) return MYEA_E_UNSUPPORTED;
  const LstmDir &D = P->d[dir];
  LstmSeq q;
  common_args(net, L, dir, q);
  q.tiles_n = static_cast<int>((P->C + PsShape<2>::BN - 1) / PsShape<2>::BN);
  q.split = PsShape<2>::SPLIT;
  q.num_kb = static_cast<int>(P->G / PS_BK);
  q.kb_per = (q.num_kb + q.split - 1) / q.split;
  q.kpa = P->dg_pan.pitch;
  q.a0 = P->dg_pan.rows.h0; q.a1 = P->dg_pan.rows.h1;
  q.a_scale = P->dg_scale;
  q.w_scale = P->w_rec_scale[dir] + P->G;
  q.act = D.act; q.cstate = D.cstate; q.cact = D.cact;
  q.deriv = L.deriv + dir * P->C;
  q.dgates = D.dgates; q.dcstate = D.dcstate;
  return launch<2>(net, q, P->G, P->w_rec[dir]);
}

}  // namespace myea

// Diagnostic (not part of the training interface): how many clusters of the two persistent kernels the device holds at
// once; a layer runs persistently when its tiles fit (see lstm_persistent_plan).
extern "C" int myea_b200_lstm_resident_clusters(int device, int *forward_pairs, int *backward_quads) {
  if (cudaSetDevice(device) != cudaSuccess) return MYEA_E_CUDA;
  if (forward_pairs) *forward_pairs = myea::resident_clusters<1>(device);
  if (backward_quads) *backward_quads = myea::resident_clusters<2>(device);
  return MYEA_OK;
}

// For tests: the barrier in front of step `step` (1 to T - 1; 0: none) of every walk in one launch of this handle is never reached, and
// the wait there gives up after `cycles` SM clocks (of a walk with resident weights so does any other wait).  MYEA_E_UNSUPPORTED when no
// layer has a walk that waits.
extern "C" int myea_b200_lstm_stall(myea_handle net, int step, uint64_t cycles) {
  if (net == nullptr || step < 0 || cycles > (1ull << 31)) return MYEA_E_INVALID;
  int found = 0;
  for (auto &L : net->layers) {
    if (L.lstm == nullptr) continue;
    if (myea::lstm_resident_stall(L.lstm, step, static_cast<long long>(cycles))) ++found;
    if (!myea::lstm_persistent_ready(L.lstm)) continue;
    L.lstm->persist->stall_step = step;
    L.lstm->persist->wait_cycles = static_cast<long long>(cycles);
    ++found;
  }
  return found > 0 ? MYEA_OK : MYEA_E_UNSUPPORTED;
}
