// All time steps of an LSTM layer in one launch with the recurrent weights RESIDENT in shared memory: networks whose batch
// is small or whose width fits few SMs, any width.
//
// The tensor-core walk (lstm_persistent.cu) streams the recurrent weight panels of a layer from L2 in every step (33 MB for
// 1024 cells) and computes tiles of 128 batch rows, however few there are; layers it does not take (widths that are no
// multiple of 8) paid three launches per time step.  With few rows a step is a matrix-vector product: every weight is used
// a handful of times, so what counts is where the weights are, and the latency of handing h (or the gate errors) to the
// next step.  4 C^2 fp32 weights fit the shared memories of the chip up to C = 1300.
//
//   groups    a group of G CTAs (one per SM) owns some rows of the batch and walks their time steps on its own; its CTAs
//             split the cells of the layer (forward: the four gate sums of cpc cells, K = C; backward: the error on h of
//             cpc cells, K = 4 C gate errors).  Both directions of a bidirectional layer run side by side.
//   step      the group's exchange buffer [K][rows] of the step before comes from L2 (G = 1: stays in shared memory), fp32
//             FMAs on 4 outputs x 4 rows per thread (one 128-bit weight read and one 128-bit input read per 16 FMAs: bound
//             by shared-memory reads at 80 % of the FMA rate), K spread over the lanes and warps of the CTA and added up in a
//             fixed order, then one thread per (row, cell) does the cell arithmetic in fp32 as lstm_cell_forward_kernel /
//             lstm_cell_backward_kernel do, leaves its result in the other exchange buffer and the group meets at a counter
//             in global memory (release / acquire, about 1 us).
//   clusters  where a group is one thread-block cluster the results go straight into the shared memories of its CTAs (st.async, 16
//             bytes of four rows each; a barrier per buffer counts the bytes of all CTAs): no counter, no trip to L2 and back, one
//             __syncthreads per step (150 cells, 50 rows, clusters of 8: forward 3.4 -> 2.5, backward 3.7 -> 2.7 us per step)
//   waits     every wait is bounded (about a second of SM clock) and raises the handle's error flag and an abort word; the
//             launch over global memory is cooperative, so all CTAs are resident (clusters are by themselves).
#include "lstm.cuh"
#include "panel_math.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace myea {

constexpr int LR_THREADS = 512, LR_WARPS = LR_THREADS / 32;
constexpr int LR_SMEM_MAX = 225 * 1024;

struct ResidentDir {
  const float *w = nullptr;      // first block of the direction in the parameter buffer
  const float *gates_in = nullptr;
  float *act = nullptr, *cstate = nullptr, *cact = nullptr, *values = nullptr;
  const uint8_t *zone_state = nullptr, *zone_output = nullptr;
  float *deriv = nullptr, *dgates = nullptr, *dcstate = nullptr;
};
struct ResidentArgs {
  int T = 0, B = 0, C = 0;
  int G = 1, groups = 1, R = 0, Rp = 0;   // CTAs per group, groups per direction, rows per group, the same rounded up to 4
  bool cluster = false;                   // a group is one cluster
  int cpc = 0, NOp = 0, K = 0;            // cells per CTA, outputs per CTA (padded to 4), length of the products
  int RB = 0, KC = 0, KW = 1;             // rows per pass, K per chunk of exchange data, warps that share an output's K range
  int RT = 4;                             // rows per thread of the products: 4 or 8
  int in_floats = 0, red_floats = 0;      // exchange data of a step (or two chunks of it) and partial sums in shared memory
  long long stride = 0, ldh = 0;
  long long rec[4] = {0, 0, 0, 0}, peep = 0;  // offsets inside a block: recurrent rows of z, i, f, o and the peepholes
  ResidentDir d[2];
  float *ex = nullptr;                    // [2 buffers][direction][group][K][Rp]
  unsigned int *sync = nullptr;           // [direction][group] counters, then one abort word
  int sync_count = 0;
  int *error_flag = nullptr;
  int stall_step = 0;                     // tests only: the step whose wait is never over (0: none); in a cluster for its first CTA
  long long wait_cycles = 1ll << 31;
};

__device__ __forceinline__ unsigned int lr_ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void lr_add_release(unsigned int *p) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }

// one thread: until the counter has reached `target`
__device__ __forceinline__ bool lr_wait(const unsigned int *counter, unsigned int target, unsigned int *abort_word, long long cycles) {
  if (lr_ld_acquire(counter) >= target) return true;
  const long long t0 = clock64();
  for (int n = 0;; ++n) {
    if (lr_ld_acquire(counter) >= target) return true;
    if ((n & 63) == 63 && (lr_ld_acquire(abort_word) != 0u || clock64() - t0 > cycles)) return false;
  }
}

__device__ __forceinline__ void lr_copy16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}

// bytes of a step's exchange data that the CTAs of a cluster push into each of them, all of them or those of CTA g
template <int KIND> __device__ __forceinline__ uint32_t lr_pushed_bytes(const ResidentArgs &q) { return static_cast<uint32_t>(q.K) * q.Rp * 4u; }
template <int KIND> __device__ __forceinline__ uint32_t lr_pushed_bytes(const ResidentArgs &q, int g) {
  return static_cast<uint32_t>(max(0, min(q.cpc, q.C - g * q.cpc))) * (KIND == 1 ? 1u : 4u) * q.Rp * 4u;
}

// One warp's share of a pass's products: RT rows x 4 outputs per thread, K in four slices over the lanes and KW over the warps.
// Lane slice ks keeps rows ks * RT / 4 ...: they go to red_s[kw][row][NOp].
template <int RT>
__device__ __forceinline__ void lr_product(float (&acc)[8][4], const float *w, int w_step, const float *x, int x_step, int trips) {
#pragma unroll 4
  for (int i = 0; i < trips; ++i, w += w_step, x += x_step) {
    const float4 wv = *reinterpret_cast<const float4 *>(w);
    const float wo[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
    for (int r4 = 0; r4 < RT; r4 += 4) {
      const float4 xv = *reinterpret_cast<const float4 *>(x + r4);
      const float xr[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int o = 0; o < 4; ++o) acc[r4 + r][o] = fmaf(xr[r], wo[o], acc[r4 + r][o]);
    }
  }
}
template <int RT>
__device__ __forceinline__ void lr_leave_sums(const float (&acc)[8][4], int lane, bool store, float *to, int pitch) {
  const int ks = lane >> 3;
  const bool up = (ks & 2) != 0, odd = (ks & 1) != 0;
  float half[RT / 2][4];
#pragma unroll
  for (int r = 0; r < RT / 2; ++r)
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const float keep = up ? acc[RT / 2 + r][o] : acc[r][o], give = up ? acc[r][o] : acc[RT / 2 + r][o];
      half[r][o] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
  for (int r = 0; r < RT / 4; ++r) {
    float mine[4];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const float keep = odd ? half[RT / 4 + r][o] : half[r][o], give = odd ? half[r][o] : half[RT / 4 + r][o];
      mine[o] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
    if (store) *reinterpret_cast<float4 *>(to + (ks * (RT / 4) + r) * pitch) = make_float4(mine[0], mine[1], mine[2], mine[3]);
  }
}

// what a cell reads from earlier launches in a step, what it takes over from its own step before (forward c and h; backward di, df,
// dc and f), and what it leaves (forward the gates, c, tanh c, h; backward the gate errors, the error on c and that on h)
struct LrIn {
  float g[4], a, dh, cp;
  bool zs, zo;
};
struct LrPeepholes {
  float i, f, o;
};
template <int KIND>
__device__ __forceinline__ void lr_cell(const LrIn &in, const LrPeepholes &p, const float (&r4)[4], bool has_rec, bool has_before, float (&kept)[4], float (&out)[7]) {
  if constexpr (KIND == 1) {
    const float cp = kept[0];
    const float z = tanh_cell(in.g[0] + r4[0]);
    const float ig = sigmoid_cell(in.g[1] + (has_rec ? r4[1] + p.i * cp : 0.f));
    const float f = sigmoid_cell(in.g[2] + r4[2] + p.f * cp), fg = has_rec ? f : 0.f;
    float cs = z * ig;
    if (has_rec) cs += fg * cp;
    if (!in.zs) cs = cp;
    const float a = tanh_cell(cs);
    const float og = sigmoid_cell(in.g[3] + r4[3] + p.o * cs);
    float h = a * og;
    if (!in.zo) h = kept[1];
    kept[0] = cs;
    kept[1] = h;
    out[0] = z; out[1] = ig; out[2] = fg; out[3] = og; out[4] = cs; out[5] = a; out[6] = h;
  } else {
    const float dh = in.dh + r4[0];
    const float z = in.g[0], ig = in.g[1], fg = in.g[2], og = in.g[3];
    const float d_o = og * (1.f - og) * (dh * in.a);
    float dc = dh * og * (1.f - in.a * in.a);
    dc += p.o * d_o;
    if (has_rec) {
      dc += p.i * kept[0];
      dc += p.f * kept[1];
      dc += kept[2] * kept[3];
    }
    const float dz = dc * ig * (1.f - z * z);
    const float di = (dc * z) * (ig * (1.f - ig));
    const float df = has_before ? (dc * in.cp) * (fg * (1.f - fg)) : 0.f;   // (the walk ends at the direction's first step)
    kept[0] = di;
    kept[1] = df;
    kept[2] = dc;
    kept[3] = fg;
    out[0] = dz; out[1] = di; out[2] = df; out[3] = d_o; out[4] = dc; out[5] = dh; out[6] = 0.f;
  }
}

// KIND 1: forward, 2: backward.  CLUSTER: the CTAs of a group are one cluster
template <int KIND, bool CLUSTER>
__global__ void __launch_bounds__(LR_THREADS, 1) lstm_resident_kernel(const __grid_constant__ ResidentArgs q) {
  extern __shared__ __align__(16) float lr_smem[];
  __shared__ volatile int s_ok[2];             // of even and odd steps: a wait of the next step may give up before every thread has read this step's
  __shared__ uint64_t landed[2];      // CLUSTER: the exchange data of a step is complete in in_s[step & 1]
  __shared__ uint32_t pushed_steps;   // CLUSTER: steps whose results this CTA has pushed
  float *red_s = lr_smem;                                // [KW][RB][NOp]
  float *w_s = lr_smem + q.red_floats;                   // [K][NOp]
  float *in_s = w_s + static_cast<size_t>(q.K) * q.NOp;  // G == 1 or a cluster: [2][K][Rp]; else one or two chunks [KC][RB]
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int per_dir = q.groups * q.G;
  const int dir = static_cast<int>(blockIdx.x) / per_dir, in_dir = static_cast<int>(blockIdx.x) - dir * per_dir;
  const int group = in_dir / q.G, g = in_dir - group * q.G;
  const ResidentDir &D = q.d[dir];
  const int cell0 = g * q.cpc, ncell = max(0, min(q.cpc, q.C - cell0));
  const int row0 = group * q.R, nrow = max(0, min(q.R, q.B - row0));
  unsigned int *counter = q.sync + dir * q.groups + group, *abort_word = q.sync + q.sync_count;
  const size_t ex_size = static_cast<size_t>(q.K) * q.Rp;
  // exchange data of even steps, and how far behind them that of odd steps lies
  const bool on_chip = CLUSTER || q.G == 1;
  float *const ex = on_chip ? in_s : q.ex + (static_cast<size_t>(dir) * q.groups + group) * ex_size;
  const size_t ex_odd = on_chip ? ex_size : static_cast<size_t>(q.sync_count) * ex_size;
  grid_dependency_wait();

  // This CTA's weights: forward [k][4 * cell + gate], backward [gate * C + k][cell].  A walk of a few steps is hardly longer than this,
  // so no element has a division of its own, and forward a lane stores the four gates of one k and cell at once: four cells and two k
  // side by side fall on different banks, where 32 k of one gate fell on two
  // (forward passes of two steps: 150 cells 23.5 -> 20.6 us, 256 36.7 -> 23.8, twice 224 48.4 -> 28.6).
  if (KIND == 1) {
    const int k_blocks = (q.C + 7) / 8, blocks = k_blocks * ((q.cpc + 3) / 4);
#pragma unroll 4
    for (int t = warp; t < blocks; t += LR_WARPS) {
      const int cb = t / k_blocks, k = (t - cb * k_blocks) * 8 + (lane >> 2), c = cb * 4 + (lane & 3);
      if (k < q.C && c < q.cpc) {
        const float *from = D.w + (cell0 + c) * q.stride + k;
        *reinterpret_cast<float4 *>(w_s + k * q.NOp + 4 * c) =
            c < ncell ? make_float4(from[q.rec[0]], from[q.rec[1]], from[q.rec[2]], from[q.rec[3]]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  } else {
    const int more_c = LR_THREADS % q.NOp, more_k = LR_THREADS / q.NOp;
    int c = tid % q.NOp, k = tid / q.NOp, gate = k / q.C;
    k -= gate * q.C;
#pragma unroll 8
    for (int i = tid; i < q.K * q.NOp; i += LR_THREADS) {
      const long long rec = gate == 0 ? q.rec[0] : gate == 1 ? q.rec[1] : gate == 2 ? q.rec[2] : q.rec[3];
      w_s[i] = c < ncell ? D.w[k * q.stride + rec + cell0 + c] : 0.f;
      c += more_c;
      k += more_k;
      if (c >= q.NOp) { c -= q.NOp; ++k; }
      while (k >= q.C) { k -= q.C; ++gate; }
    }
  }
  if (!CLUSTER && q.G == 1)
    for (int i = tid; i < static_cast<int>(2 * ex_size); i += LR_THREADS) in_s[i] = 0.f;
  if (tid == 0) {
    s_ok[0] = s_ok[1] = 1;
    if constexpr (CLUSTER) {
      ptx::mbar_init(&landed[0], 1);
      ptx::mbar_init(&landed[1], 1);
      ptx::fence_barrier_init();
      for (int s = 0; s < min(2, q.T - 1); ++s) ptx::mbar_arrive_expect_tx(&landed[s], lr_pushed_bytes<KIND>(q));
    }
  }
  __syncthreads();
  if constexpr (CLUSTER) ptx::cluster_sync_all();

  const int tiles_c = (q.NOp / 4 + 7) / 8, row_tiles = q.RB / q.RT;
  const int kw = warp % q.KW, my_task = warp / q.KW;
  const int tile_c = my_task % tiles_c, tile_r = my_task / tiles_c;
  const bool has_task = tile_r < row_tiles;
  const int col = min(tile_c * 8 + (lane & 7), q.NOp / 4 - 1) * 4;   // first of this thread's four outputs
  const bool col_live = tile_c * 8 + (lane & 7) < q.NOp / 4;
  const int task_row = tile_r * q.RT, k_first = kw * 4 + (lane >> 3), k_step = 4 * q.KW;
  auto trips = [&](int n) { return n > k_first ? (n - k_first + k_step - 1) / k_step : 0; };
  const float *const w_mine = w_s + static_cast<size_t>(k_first) * q.NOp + col;
  float *const sums_mine = red_s + (static_cast<size_t>(kw) * q.RB + task_row) * q.NOp + col;
  const int w_step = k_step * q.NOp, all_trips = trips(q.K);
  const int chunks = on_chip ? 1 : (q.K + q.KC - 1) / q.KC, buffers = chunks > 1 ? 2 : 1;
  const bool reverse = dir != 0;
  const long long C = q.C;

  // One thread per (row, cell).  CLUSTER: four neighbouring lanes are four rows of one cell.
  auto row_of = [&](int u) { return CLUSTER ? u / (4 * ncell) * 4 + (u & 3) : u / ncell; };
  auto cell_of = [&](int u) { return CLUSTER ? (u >> 2) % ncell : u % ncell; };
  const int my_row = row_of(tid), my_cell = cell_of(tid);
  const bool upwards = (KIND == 1) != reverse;   // forward: step s of the direction; backward: the walk goes against it
  auto time_of = [&](int s) { return upwards ? s : q.T - 1 - s; };
  const long long dc_step = (upwards ? 1 : -1) * static_cast<long long>(q.B) * C, dh_step = (upwards ? 1 : -1) * static_cast<long long>(q.B) * q.ldh;
  auto load_peepholes = [&](int c) {
    const float *p = D.w + (cell0 + c) * q.stride + q.peep;
    return LrPeepholes{p[0], p[1], p[2]};
  };
  // Where a step's arrays lie for one row and cell: [T][B][4C] read (gate inputs; gates) and left (gates; gate errors), [T][B][C] and
  // [T][B][ldh]
  struct Places {
    const float *g4;
    float *left4, *c, *a, *h;
    const uint8_t *zs, *zo;
  };
  auto places = [&](int s, int rg, int c) {
    const long long t = time_of(s), row = t * q.B + row0 + rg, cell = cell0 + c;
    Places x;
    x.g4 = (KIND == 1 ? D.gates_in : D.act) + row * 4 * C + cell;
    x.left4 = (KIND == 1 ? D.act : D.dgates) + row * 4 * C + cell;
    x.c = (KIND == 1 ? D.cstate : D.dcstate) + row * C + cell;
    x.a = D.cact + row * C + cell;
    x.h = (KIND == 1 ? D.values : D.deriv) + row * q.ldh + cell;
    x.zs = KIND == 1 && D.zone_state != nullptr ? D.zone_state + t * C + cell : nullptr;
    x.zo = KIND == 1 && D.zone_output != nullptr ? D.zone_output + t * C + cell : nullptr;
    return x;
  };
  auto load = [&](const Places &x, const float *c_before, LrIn &in) {
#pragma unroll
    for (int k = 0; k < 4; ++k) in.g[k] = x.g4[k * C];
    if constexpr (KIND == 1) {
      in.zs = x.zs == nullptr || *x.zs != 0;
      in.zo = x.zo == nullptr || *x.zo != 0;
    } else {
      in.a = *x.a;
      in.dh = *x.h;
      in.cp = c_before != nullptr ? *c_before : 0.f;
    }
  };
  auto leave = [&](const Places &x, const float (&out)[7], bool has_rec) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x.left4[k * C] = out[k];
    *x.c = out[4];
    if constexpr (KIND == 1) {
      *x.a = out[5];
      *x.h = out[6];
    } else if (has_rec) {
      *x.h = out[5];
    }
  };
  // A thread that has the same row and cell in every step keeps its places and what it passes on to the next one, and fetches that
  // one's arrays a step ahead: they come from memory, and a step is hardly longer than the way there.  (The arrays' pointers lie
  // in the kernel's arguments, indexed by the direction: fetching them anew was a good part of a step.)
  const bool early = q.RB == q.Rp && q.Rp * ncell <= LR_THREADS;
  const bool mine = early && tid < q.Rp * ncell && my_row < nrow;
  LrPeepholes peep = {0.f, 0.f, 0.f};
  LrIn ahead = {};
  Places at = {};
  const float *c_before = nullptr;   // backward: the cell state of the time before
  if (mine) {
    peep = load_peepholes(my_cell);
    at = places(0, my_row, my_cell);
    if (KIND == 2 && q.T > 1) c_before = D.cstate + (static_cast<long long>(time_of(1)) * q.B + row0 + my_row) * C + cell0 + my_cell;
    load(at, c_before, ahead);
  }
  float kept[4] = {0.f, 0.f, 0.f, 0.f};
  // CLUSTER (of up to 8): CTAs lane & 3 and that + 4 get what this lane's quad pushes
  const uint32_t base = ptx::smem_u32(lr_smem), landed_at = ptx::smem_u32(&landed[0]) - base;
  uint32_t peer[2] = {};
  if constexpr (CLUSTER) {
#pragma unroll
    for (int j = 0; j < 2; ++j) peer[j] = ptx::map_to_cta(base, static_cast<uint32_t>(min((lane & 3) + 4 * j, q.G - 1)));
  }

  int s = 0;
  bool ok = true;
  for (; s < q.T; ++s) {
    const bool has_rec = s > 0;
    if (CLUSTER && has_rec) {
      // (every thread waits by itself; what it reads after a wait that gave up is not used: s_ok below)
      uint64_t *bar = &landed[(s - 1) & 1];
      const uint32_t parity = static_cast<uint32_t>((s - 1) >> 1) & 1u;
      const bool stalled = s == q.stall_step && g == 0;   // (s is 1 at least here)
      if (stalled || !ptx::mbar_try_wait_acquire_cluster(bar, parity)) {
        const long long t0 = clock64();
        while (stalled || !ptx::mbar_try_wait_acquire_cluster(bar, parity)) {
          if (clock64() - t0 > q.wait_cycles) {
            s_ok[s & 1] = 0;
            atomicCAS(q.error_flag, 0, 412);
            break;
          }
        }
      }
    } else if (has_rec && q.G > 1) {
      if (tid == 0 && !lr_wait(counter, static_cast<unsigned int>(q.G) * static_cast<unsigned int>(s) + (s == q.stall_step ? 1u : 0u), abort_word, q.wait_cycles)) {
        s_ok[s & 1] = 0;
        atomicCAS(q.error_flag, 0, 411);
        atomicExch(abort_word, 1u);
      }
      __syncthreads();
      ok = s_ok[s & 1] != 0;
      if (!ok) break;
    }
    const size_t src_at = (s & 1) != 0 ? 0 : ex_odd, dst_at = (s & 1) != 0 ? ex_odd : 0;
    for (int rb = 0; rb < q.Rp; rb += q.RB) {
      const int rows_here = min(q.RB, q.Rp - rb);
      if (has_rec) {
        float acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int o = 0; o < 4; ++o) acc[r][o] = 0.f;
        const bool works = has_task && task_row < rows_here;
        auto multiply = [&](const float *w, const float *x, int pitch, int n) {
          if (!works) return;
          x += k_first * pitch + task_row;
          if (q.RT == 8) lr_product<8>(acc, w, w_step, x, k_step * pitch, n);
          else lr_product<4>(acc, w, w_step, x, k_step * pitch, n);
        };
        if (on_chip) {
          multiply(w_mine, in_s + src_at + rb, q.Rp, all_trips);
        } else {
          // (every CTA of a group reads the same data: each starts at a place of its own)
          const int groups4 = rows_here / 4;
          const float *src = ex + src_at;
          auto fetch = [&](int ch) {
            const int k0 = ch * q.KC, n = min(q.KC, q.K - k0) * groups4, first = static_cast<int>(static_cast<long long>(n) * g / q.G);
            float *to = in_s + (ch % buffers) * q.KC * q.RB;
            for (int i = tid; i < n; i += LR_THREADS) {
              int j = i + first;
              if (j >= n) j -= n;
              const int k = j / groups4, r = (j - k * groups4) * 4;
              lr_copy16(to + k * q.RB + r, src + static_cast<size_t>(k0 + k) * q.Rp + rb + r);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
          };
          fetch(0);
          for (int ch = 0; ch < chunks; ++ch) {
            if (ch + 1 < chunks) {
              fetch(ch + 1);
              asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
              asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            multiply(w_mine + static_cast<size_t>(ch) * q.KC * q.NOp, in_s + (ch % buffers) * q.KC * q.RB, q.RB, trips(min(q.KC, q.K - ch * q.KC)));
            if (ch + 1 < chunks) __syncthreads();   // the buffer is refilled by the next but one fetch
          }
        }
        if (q.RT == 8) lr_leave_sums<8>(acc, lane, works && col_live, sums_mine, q.NOp);
        else lr_leave_sums<4>(acc, lane, works && col_live, sums_mine, q.NOp);
        __syncthreads();
        if constexpr (CLUSTER) {
          ok = s_ok[s & 1] != 0;
          if (!ok) break;
          if (rb == 0 && tid == 0 && s + 2 < q.T) ptx::mbar_arrive_expect_tx(&landed[(s + 1) & 1], lr_pushed_bytes<KIND>(q));   // of step s + 1
        }
      }
      // the recurrent sums of one (row, cell)
      auto recurrent = [&](int rl, int c, float (&r4)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) r4[k] = 0.f;
        if (!has_rec) return;
        const float *p = red_s + static_cast<size_t>(rl) * q.NOp + (KIND == 1 ? 4 * c : c);
        const int pitch = q.RB * q.NOp;
#pragma unroll 4
        for (int k = 0; k < q.KW; ++k, p += pitch) {
          if constexpr (KIND == 1) {
            const float4 v = *reinterpret_cast<const float4 *>(p);
            r4[0] += v.x; r4[1] += v.y; r4[2] += v.z; r4[3] += v.w;
          } else {
            r4[0] += *p;
          }
        }
      };
      // ... and what the next step reads of it: into the exchange data; CLUSTER: of four rows at a time into that of every CTA
      auto hand_on = [&](int rl, int c, bool live, const float (&out)[7]) {
        const int cell = cell0 + c;
        if constexpr (CLUSTER) {
          if (s + 1 >= q.T) return;
          const unsigned mask = 0xFu << (lane & 28);
          const uint32_t bar = landed_at + (s & 1) * 8;
          uint32_t to = ptx::smem_u32(in_s) - base + (static_cast<uint32_t>(dst_at) + static_cast<uint32_t>(cell) * q.Rp + rb + (rl & ~3)) * 4u;
#pragma unroll
          for (int k = 0; k < (KIND == 1 ? 1 : 4); ++k, to += static_cast<uint32_t>(q.C) * q.Rp * 4u) {
            const float x = live ? out[KIND == 1 ? 6 : k] : 0.f;
            const float4 v = make_float4(__shfl_sync(mask, x, lane & 28), __shfl_sync(mask, x, (lane & 28) + 1), __shfl_sync(mask, x, (lane & 28) + 2),
                                         __shfl_sync(mask, x, (lane & 28) + 3));
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if ((lane & 3) + 4 * j < q.G) ptx::st_async_f4(peer[j] + to, v, peer[j] + bar);
          }
        } else {
          float *e = ex + dst_at + static_cast<size_t>(cell) * q.Rp + rb + rl;
          if constexpr (KIND == 1) {
            *e = out[6];
          } else {
            const size_t gate_step = static_cast<size_t>(q.C) * q.Rp;
            e[0] = out[0]; e[gate_step] = out[1]; e[2 * gate_step] = out[2]; e[3 * gate_step] = out[3];
          }
        }
      };
      float out[7], r4[4];
      if (early) {
        if (tid < rows_here * ncell && (CLUSTER || my_row < nrow)) {
          const LrIn in = ahead;
          if (mine && s + 1 < q.T) {
            at.g4 += 4 * dc_step;
            if constexpr (KIND == 1) {
              if (at.zs != nullptr) at.zs += upwards ? C : -C;
              if (at.zo != nullptr) at.zo += upwards ? C : -C;
              load(at, nullptr, ahead);
            } else {
              Places next = at;
              next.a += dc_step;
              next.h += dh_step;
              c_before = s + 2 < q.T ? c_before + dc_step : nullptr;
              load(next, c_before, ahead);
            }
          }
          recurrent(my_row, my_cell, r4);
          lr_cell<KIND>(in, peep, r4, has_rec, s + 1 < q.T, kept, out);
          hand_on(my_row, my_cell, my_row < nrow, out);
        }
      } else {
        for (int u = tid; u < rows_here * ncell; u += LR_THREADS) {
          const int rl = u == tid ? my_row : row_of(u), c = u == tid ? my_cell : cell_of(u), rg = rb + rl;
          const bool live = rg < nrow;   // else padding of the row count
          if (!CLUSTER && !live) continue;
          Places x = {};
          LrIn in = {};
          LrPeepholes p = {0.f, 0.f, 0.f};
          if (live) {
            x = places(s, rg, c);
            p = load_peepholes(c);
            const float *before = KIND == 2 && s + 1 < q.T ? D.cstate + (static_cast<long long>(time_of(s + 1)) * q.B + row0 + rg) * C + cell0 + c : nullptr;
            load(x, before, in);
            if (has_rec) {
              if constexpr (KIND == 1) {
                kept[0] = *(x.c - dc_step);
                kept[1] = *(x.h - dh_step);
              } else {
                kept[0] = (x.left4 - 4 * dc_step)[C];
                kept[1] = (x.left4 - 4 * dc_step)[2 * C];
                kept[2] = *(x.c - dc_step);
                kept[3] = (x.g4 - 4 * dc_step)[2 * C];
              }
            } else {
              kept[0] = kept[1] = 0.f;
            }
          }
          recurrent(rl, c, r4);
          lr_cell<KIND>(in, p, r4, has_rec, s + 1 < q.T, kept, out);
          hand_on(rl, c, live, out);
          if (live) leave(x, out, has_rec);
        }
      }
      // red_s and (G = 1) the exchange buffer are complete / free again.  (A cluster's last pass: whoever writes red_s in the next
      // step has waited for what this CTA's cells, which read it, have pushed.)
      if (!CLUSTER || rb + q.RB < q.Rp) __syncthreads();
      if (!CLUSTER && q.G > 1 && tid == 0 && rb + q.RB >= q.Rp) lr_add_release(counter);
      if (mine) {   // what only later launches read is stored behind what the group waits for
        leave(at, out, has_rec);
        at.left4 += 4 * dc_step;
        at.c += dc_step;
        at.a += dc_step;
        at.h += dh_step;
      }
    }
    if (CLUSTER && !ok) break;
  }
  if constexpr (CLUSTER) {
    // Nobody leaves while another CTA may push into its shared memory.  All steps done: whatever was sent here has been waited
    // for.  After a wait that gave up in step s: of steps s - 1 and s, which may be on their way, what will not come is counted in
    // and the rest waited for.
    if (tid == 0) pushed_steps = static_cast<uint32_t>(s);
    __syncthreads();
    ptx::cluster_sync_all();
    if (s < q.T && tid == 0) {
      for (int x = s - 1; x <= min(s, q.T - 2); ++x) {
        uint32_t missing = 0;
        for (int g2 = 0; g2 < q.G; ++g2)
          if (ptx::ld_cluster_u32(ptx::map_to_cta(ptx::smem_u32(&pushed_steps), static_cast<uint32_t>(g2))) <= static_cast<uint32_t>(x)) missing += lr_pushed_bytes<KIND>(q, g2);
        if (missing != 0u) ptx::mbar_complete_tx(&landed[x & 1], missing);
        ptx::mbar_wait(&landed[x & 1], static_cast<uint32_t>(x >> 1) & 1u);
      }
    }
    __syncthreads();
    ptx::cluster_sync_all();
  }
}

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
struct LstmResident {
  ResidentArgs f, b;      // forward / backward launch shapes; the pointers are filled in per call
  size_t smem_f = 0, smem_b = 0;
  float *ex = nullptr;
  unsigned int *sync = nullptr;
  int stall_step = 0;     // see ResidentArgs
  long long wait_cycles = 1ll << 31;
};

// shape of one kind for G CTAs per group (one cluster or not) where `max_groups` of them run at once; false when it does not fit.
// clocks: estimate of a step
static bool resident_shape(int kind, long long B, long long C, long long max_groups, int G, bool cluster, ResidentArgs *q, size_t *smem, double *clocks) {
  const int cpc = static_cast<int>((C + G - 1) / G);
  if (static_cast<int>((C + cpc - 1) / cpc) != G) return false;
  if (max_groups < 1) return false;
  q->G = G;
  q->cluster = cluster;
  q->cpc = cpc;
  q->C = static_cast<int>(C); q->B = static_cast<int>(B);
  q->R = static_cast<int>((B + max_groups - 1) / max_groups);
  q->Rp = (q->R + 3) / 4 * 4;
  q->groups = static_cast<int>((B + q->R - 1) / q->R);
  q->K = static_cast<int>(kind == 1 ? C : 4 * C);
  q->NOp = kind == 1 ? 4 * cpc : (cpc + 3) / 4 * 4;
  const int tiles_c = (q->NOp / 4 + 7) / 8;
  if (tiles_c > LR_WARPS) return false;
  // eight rows per thread halve the reads of the weights; with few K per warp they only lengthen the sums across lanes
  q->RT = q->Rp % 8 == 0 && q->K >= 512 ? 8 : 4;
  q->RB = std::min(q->Rp, q->RT * (LR_WARPS / tiles_c));
  const int tasks = tiles_c * (q->RB / q->RT);
  q->KW = LR_WARPS / tasks;
  q->red_floats = q->KW * q->RB * q->NOp;
  // The whole exchange data of a pass where it fits: every chunk more is another trip to L2 within the step (1024 cells,
  // 16 rows: four chunks of 20 KB 11.3 us per step, one of 64 KB 9.7).
  const long long room = LR_SMEM_MAX / static_cast<long long>(sizeof(float)) - static_cast<long long>(q->K) * q->NOp - q->red_floats;
  if (G == 1 || cluster) {
    if (2ll * q->K * q->Rp > room) return false;
    q->KC = q->K;
    q->in_floats = 2 * q->K * q->Rp;
  } else if (static_cast<long long>(q->K) * q->RB <= room) {
    q->KC = q->K;
    q->in_floats = q->K * q->RB;
  } else {
    if (room / 2 / q->RB < 4 * q->KW) return false;
    q->KC = static_cast<int>(room / 2 / q->RB / (4 * q->KW)) * (4 * q->KW);
    q->in_floats = 2 * q->KC * q->RB;
  }
  *smem = (static_cast<size_t>(q->K) * q->NOp + static_cast<size_t>(q->in_floats) + q->red_floats) * sizeof(float);
  const double passes = static_cast<double>((q->Rp + q->RB - 1) / q->RB);
  const double reads = passes * tasks * (q->K / 4.0) * (4.0 + q->RT / 4.0);        // shared-memory wavefronts
  const double issue = passes * (q->K / (4.0 * q->KW)) * (4.0 + 4.0 * q->RT);      // one warp's share, instruction by instruction
  // Fitted to the clock (1.9 GHz) over the shapes below, within 20 % for most: products, exchange, and the cells, whose instructions
  // follow one another (and whose arrays are fetched late where a thread has more than one cell)
  const double bytes = q->K * static_cast<double>(q->Rp) * 4.0, chunks = (q->K + q->KC - 1) / q->KC, work = std::max(reads, issue);
  const double cells = static_cast<double>(q->Rp) * cpc * (q->RB == q->Rp && q->Rp * cpc <= LR_THREADS ? 1.0 : 2.5);
  const double forward = 500.0 + 1.05 * work + 12.0 * cells + 17.0 * q->KW + (G == 1 ? 0.0 : cluster ? 1200.0 + 77.0 * G + bytes / 5.5 : 4700.0 + bytes / 10.0);
  const double backward = 1400.0 + 0.77 * work + 5.6 * cells + (G == 1 ? 0.0 : cluster ? 1150.0 + bytes / 6.2 : 3100.0 + bytes / 9.0);
  *clocks = (kind == 1 ? forward : backward) + 900.0 * (passes - 1.0) + 1000.0 * passes * (chunks - 1.0);
  return true;
}

template <int KIND, bool CLUSTER> static bool allow_smem() {
  auto kernel = lstm_resident_kernel<KIND, CLUSTER>;
  const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LR_SMEM_MAX) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok;
}

// clusters of G CTAs, each with an SM to itself, that the device runs at once
template <int KIND> static int cluster_capacity(int sms, int G) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sms / G * G));
  cfg.blockDim = dim3(LR_THREADS);
  cfg.dynamicSmemBytes = LR_SMEM_MAX;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(G);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, lstm_resident_kernel<KIND, true>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  return n;
}

// Which walk a pass takes, measured per time step and direction (us; weights loaded, T = 72 against T = 8; resident: over global memory |
// on clusters of 8, both directions of "x 2" together):
//                     forward                                   backward
//   cells x rows      resident       tensor  launches           resident       tensor  launches
//    64 x 32           1.7 | 1.8                                 1.5 | 2.1
//   128 x 32           3.2 | 1.9      6.5                        3.4 | 2.4      6.7
//   150 x 50           3.8 | 2.6                                 3.8 | 2.7
//   150 x 50 x 2       4.4 | 3.4, on 4 3.1                       3.6 | 3.9, on 4 3.1
//   256 x 32           3.6 | 2.7                                 4.1 | 3.1
//   256 x 256          8.8           10.5                        8.9           12.9
//   301 x 32           4.5 | 3.7                                 4.5
//   301 x 200         11.3 | 15.6                               10.2
//   512 x 16           4.2            8.9                        5.5           10.1
//   601 x 128         22.1                     24.0             25.1                     25.0
//   768 x 32           9.6           10.5                       23.3           13.1
//   1001 x 32         19.9                     24.6             54.6                     34.6
//   1024 x 4           4.9           11.7                        8.3           14.9
//   1024 x 16          8.5           11.7                       28.0           14.6
//   1024 x 256       113.8           14.7                      414.6           20.8
// Backward K is four times as long and only a quarter as wide, so the two passes cross at different sizes and are chosen by
// themselves (all walks leave the same arrays).
static double resident_walk_us(double clocks) { return clocks / 1900.0; }
static double other_walk_us(const LstmPlan *P, int kind, long long B) {   // per direction: one after the other
  const double C = static_cast<double>(P->C), rows = static_cast<double>(std::min<long long>(B, 128)) / 128.0, more = B > 128 ? 0.5 : 0.0;
  if (lstm_persistent_ready(P)) return kind == 1 ? 6.2 + 5.5 * C / 1024.0 + 2.7 * rows + more : 5.0 + 9.6 * C / 1024.0 + 5.6 * rows + more;
  const double products = static_cast<double>(B) * 4.0 * C * C;   // straight from fp32 or, from 600 Mi on, from panels
  return 5.5 + 0.0148 * C + products * 2e-6 / (products <= 629145600.0 ? 36.0 : 75.0);
}

int lstm_resident_plan(myea_b200_net *net, LayerPlan &L) {
  LstmPlan *P = L.lstm;
  P->resident = nullptr;
  P->resident_pass[0] = P->resident_pass[1] = false;
  if (net->ctx.gemm_engine != 0 || P->cpb != 1 || P->C > 1400) return MYEA_OK;
  int sms = 0, coop = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->ctx.device) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, net->ctx.device) != cudaSuccess || !coop)
    return MYEA_OK;
  LstmResident best;
  double best_clocks[2] = {1e30, 1e30};
  if (!allow_smem<1, false>() || !allow_smem<2, false>() || !allow_smem<1, true>() || !allow_smem<2, true>()) return MYEA_OK;
  auto consider = [&](int G, bool cluster, long long groups_f, long long groups_b) {
    ResidentArgs q;
    size_t smem = 0;
    double c = 1e30;
    if (resident_shape(1, net->B, P->C, groups_f, G, cluster, &q, &smem, &c) && c < best_clocks[0]) { best_clocks[0] = c; best.f = q; best.smem_f = smem; }
    q = ResidentArgs();
    if (resident_shape(2, net->B, P->C, groups_b, G, cluster, &q, &smem, &c) && c < best_clocks[1]) { best_clocks[1] = c; best.b = q; best.smem_b = smem; }
  };
  for (int G = 1; G * P->dirs <= sms; ++G) consider(G, false, sms / (P->dirs * G), sms / (P->dirs * G));
  // (clusters of 16 are few: 256 cells and 32 rows 3.0 us on them against 2.7 on 8)
  for (int G = 2; G <= 8; G *= 2) consider(G, true, cluster_capacity<1>(sms, G) / P->dirs, cluster_capacity<2>(sms, G) / P->dirs);
  for (int k = 0; k < 2; ++k)
    P->resident_pass[k] = best_clocks[k] < 1e29 && resident_walk_us(best_clocks[k]) < other_walk_us(P, k + 1, net->B) * P->dirs;
  if (!P->resident_pass[0] && !P->resident_pass[1]) return MYEA_OK;
  LstmResident *r = new LstmResident(best);
  P->resident = r;
  // (a pass that is not taken here has groups, K and Rp of its best shape or of none: both only size the buffers, which the two passes
  // share.  Rows that pad a group are numbers of no use: zeros at first, then what the other pass has left there; no live row reads them)
  const int counters = P->dirs * std::max(r->f.groups, r->b.groups);
  void *p = nullptr;
  const size_t ex_floats = 2 * static_cast<size_t>(P->dirs) * std::max(static_cast<size_t>(r->f.groups) * r->f.K * r->f.Rp, static_cast<size_t>(r->b.groups) * r->b.K * r->b.Rp);
  if (cudaMalloc(&p, ex_floats * sizeof(float)) != cudaSuccess) { net->ctx.error = "cudaMalloc failed (LSTM exchange buffer)"; return MYEA_E_CUDA; }
  net->allocations.push_back(p);
  r->ex = static_cast<float *>(p);
  if (cudaMemsetAsync(p, 0, ex_floats * sizeof(float), net->ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  if (cudaMalloc(&p, (counters + 1) * sizeof(unsigned int)) != cudaSuccess) { net->ctx.error = "cudaMalloc failed (LSTM step counters)"; return MYEA_E_CUDA; }
  net->allocations.push_back(p);
  r->sync = static_cast<unsigned int *>(p);
  return MYEA_OK;
}

// Tests: see myea_b200_lstm_stall.  False where no CTA of this layer's walks waits for another.
bool lstm_resident_stall(LstmPlan *P, int step, long long cycles) {
  if (P->resident == nullptr) return false;
  P->resident->stall_step = step;
  P->resident->wait_cycles = cycles;
  return (P->resident_pass[0] && P->resident->f.G > 1) || (P->resident_pass[1] && P->resident->b.G > 1);
}

void lstm_resident_destroy(LstmPlan *P) {
  if (P != nullptr) { delete P->resident; P->resident = nullptr; }
}

// runs every direction of the layer: kind 1 forward (gates_in is complete), 2 backward (deriv holds the error from above)
int lstm_resident_run(myea_b200_net *net, LayerPlan &L, int kind, bool zoneout, const long long rec[4], long long peep) {
  LstmPlan *P = L.lstm;
  LstmResident *r = P->resident;
  Context &ctx = net->ctx;
  ResidentArgs q = kind == 1 ? r->f : r->b;
  q.T = static_cast<int>(net->T);
  q.stride = P->stride;
  q.ldh = L.n_out;
  for (int g = 0; g < 4; ++g) q.rec[g] = rec[g];
  q.peep = peep;
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    ResidentDir &o = q.d[d];
    o.w = net->params + D.w_base;
    o.gates_in = D.gates_in; o.act = D.act; o.cstate = D.cstate; o.cact = D.cact;
    o.values = L.values + d * P->C;
    o.zone_state = zoneout ? D.zone_state : nullptr;
    o.zone_output = zoneout ? D.zone_output : nullptr;
    o.deriv = L.deriv + d * P->C;
    o.dgates = D.dgates; o.dcstate = D.dcstate;
  }
  q.ex = r->ex;
  q.sync = r->sync;
  q.sync_count = P->dirs * q.groups;
  q.error_flag = ctx.d_error_flag;
  q.stall_step = r->stall_step;
  q.wait_cycles = r->wait_cycles;
  if (q.G > 1 && !q.cluster && cudaMemsetAsync(q.sync, 0, (q.sync_count + 1) * sizeof(unsigned int), ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(P->dirs * q.groups * q.G));
  cfg.blockDim = dim3(LR_THREADS);
  cfg.dynamicSmemBytes = kind == 1 ? r->smem_f : r->smem_b;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (q.cluster) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(q.G);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = (ctx.dependent_launch && !ctx.profiling) ? 1 : 0;
    cfg.numAttrs = 2;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  auto kernel = kind == 1 ? (q.cluster ? lstm_resident_kernel<1, true> : lstm_resident_kernel<1, false>)
                          : (q.cluster ? lstm_resident_kernel<2, true> : lstm_resident_kernel<2, false>);
  ctx.begin(TC_RECURRENT);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, q);
  ctx.end(TC_RECURRENT);
  ctx.gemm_flops += P->dirs * 2.0 * q.B * 4.0 * q.C * q.C * (q.T - 1);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

}  // namespace myea

// For tests: the walk that pass `kind` (1 forward, 2 backward) of layer `layer` takes.  walk: 0 launches, 1 tensor cores, 2 resident weights; of
// the latter: CTAs per group, whether they are a cluster, groups per direction, row passes per step, rows per thread, whether a thread keeps one
// row and cell.
extern "C" int myea_b200_lstm_walk(myea_handle net, uint32_t layer, int kind, int out[7]) {
  if (net == nullptr || out == nullptr || layer >= net->layers.size() || (kind != 1 && kind != 2)) return MYEA_E_INVALID;
  const myea::LstmPlan *P = net->layers[layer].lstm;
  if (P == nullptr || P->cpb != 1) return MYEA_E_INVALID;
  for (int i = 0; i < 7; ++i) out[i] = 0;
  if (!P->resident_pass[kind - 1]) {
    out[0] = myea::lstm_persistent_ready(P) ? 1 : 0;
    return MYEA_OK;
  }
  const myea::ResidentArgs &q = kind == 1 ? P->resident->f : P->resident->b;
  out[0] = 2;
  out[1] = q.G;
  out[2] = q.cluster ? 1 : 0;
  out[3] = q.groups;
  out[4] = (q.Rp + q.RB - 1) / q.RB;
  out[5] = q.RT;
  out[6] = q.RB == q.Rp && q.Rp * q.cpc <= myea::LR_THREADS ? 1 : 0;
  return MYEA_OK;
}
