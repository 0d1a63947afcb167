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
//   waits     every wait is bounded (about a second of SM clock) and raises the handle's error flag and an abort word; the
//             launch is cooperative, so all CTAs are resident.
#include "lstm.cuh"
#include "panel_math.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace myea {

constexpr int LR_THREADS = 512, LR_WARPS = LR_THREADS / 32;
constexpr int LR_RED_FLOATS = 4 * LR_WARPS * 32;     // partial sums: KW * RB * NOp floats, 4 rows x 32 outputs per warp at most
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
  int cpc = 0, NOp = 0, K = 0;            // cells per CTA, outputs per CTA (padded to 4), length of the products
  int RB = 0, KC = 0, KW = 1;             // rows per pass, K per chunk of exchange data, warps that share an output's K range
  int in_floats = 0;                      // exchange data of a step (or two chunks of it) in shared memory
  long long stride = 0, ldh = 0;
  long long rec[4] = {0, 0, 0, 0}, peep = 0;  // offsets inside a block: recurrent rows of z, i, f, o and the peepholes
  ResidentDir d[2];
  float *ex = nullptr;                    // [2 buffers][direction][group][K][Rp]
  unsigned int *sync = nullptr;           // [direction][group] counters, then one abort word
  int sync_count = 0;
  int *error_flag = nullptr;
};

__device__ __forceinline__ unsigned int lr_ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void lr_add_release(unsigned int *p) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }

// one thread: until the counter has reached `target`
__device__ __forceinline__ bool lr_wait(const unsigned int *counter, unsigned int target, unsigned int *abort_word) {
  if (lr_ld_acquire(counter) >= target) return true;
  const long long t0 = clock64();
  for (int n = 0;; ++n) {
    if (lr_ld_acquire(counter) >= target) return true;
    if ((n & 63) == 63 && (lr_ld_acquire(abort_word) != 0u || clock64() - t0 > (1ll << 31))) return false;
  }
}

__device__ __forceinline__ void lr_copy16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}

// KIND 1: forward, 2: backward
template <int KIND>
__global__ void __launch_bounds__(LR_THREADS, 1) lstm_resident_kernel(const __grid_constant__ ResidentArgs q) {
  extern __shared__ __align__(16) float lr_smem[];
  __shared__ int s_ok;
  float *red_s = lr_smem;                                // [KW][RB][NOp]
  float *w_s = lr_smem + LR_RED_FLOATS;                  // [K][NOp]
  float *in_s = w_s + static_cast<size_t>(q.K) * q.NOp;  // G == 1: [2][K][Rp]; else one or two chunks [KC][RB]
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int per_dir = q.groups * q.G;
  const int dir = static_cast<int>(blockIdx.x) / per_dir, in_dir = static_cast<int>(blockIdx.x) - dir * per_dir;
  const int group = in_dir / q.G, g = in_dir - group * q.G;
  const ResidentDir &D = q.d[dir];
  const int cell0 = g * q.cpc, ncell = max(0, min(q.cpc, q.C - cell0));
  const int row0 = group * q.R, nrow = max(0, min(q.R, q.B - row0));
  unsigned int *counter = q.sync + dir * q.groups + group, *abort_word = q.sync + q.sync_count;
  const size_t ex_size = static_cast<size_t>(q.K) * q.Rp;
  float *ex[2];
#pragma unroll
  for (int b = 0; b < 2; ++b)
    ex[b] = q.G == 1 ? in_s + b * ex_size : q.ex + (static_cast<size_t>(b) * q.sync_count + dir * q.groups + group) * ex_size;
  grid_dependency_wait();

  // this CTA's weights: forward [k][4 * cell + gate], backward [gate * C + k][cell]
  if (KIND == 1) {
#pragma unroll 8
    for (int i = tid; i < q.cpc * 4 * q.C; i += LR_THREADS) {
      const int k = i % q.C, o = i / q.C, c = o >> 2;
      w_s[k * q.NOp + o] = c < ncell ? D.w[(cell0 + c) * q.stride + q.rec[o & 3] + k] : 0.f;
    }
  } else {
#pragma unroll 8
    for (int i = tid; i < q.K * q.NOp; i += LR_THREADS) {
      const int c = i % q.NOp, kk = i / q.NOp, gate = kk / q.C, k = kk - gate * q.C;
      w_s[i] = c < ncell ? D.w[k * q.stride + q.rec[gate] + cell0 + c] : 0.f;
    }
  }
  if (q.G == 1)
    for (int i = tid; i < static_cast<int>(2 * ex_size); i += LR_THREADS) in_s[i] = 0.f;
  if (tid == 0) s_ok = 1;
  __syncthreads();

  const int tiles_c = (q.NOp / 4 + 7) / 8, row_tiles = q.RB / 4;
  const int kw = warp % q.KW, my_task = warp / q.KW;
  const int tile_c = my_task % tiles_c, tile_r = my_task / tiles_c;
  const bool has_task = tile_r < row_tiles;
  const int ks = lane >> 3;
  const int col = min(tile_c * 8 + (lane & 7), q.NOp / 4 - 1) * 4;   // first of this thread's four outputs
  const bool col_live = tile_c * 8 + (lane & 7) < q.NOp / 4;
  const bool reverse = dir != 0;

  for (int s = 0; s < q.T; ++s) {
    // forward: step s of the direction; backward: the walk goes against it
    const int t = (KIND == 1) != reverse ? s : q.T - 1 - s;
    const bool later_is_plus = !reverse;                       // whether time t + 1 is the later step of the direction
    const int tp = later_is_plus ? t - 1 : t + 1, tn = later_is_plus ? t + 1 : t - 1;
    const bool has_rec = s > 0;
    // what the cell arithmetic reads besides the sums (all of it from earlier launches or written by this same thread): where a
    // thread has one (row, cell) per step it is fetched before the wait for the group
    struct {
      float g[4], p_i, p_f, p_o, cp, hp, a, dh, dni, dnf, dcn, fn;
      bool zs, zo;
    } in;
    const long long C = q.C;
    auto load = [&](int rg, int c) {
      const long long b = row0 + rg, cell = cell0 + c;
      const long long at = static_cast<long long>(t) * q.B + b, atp = static_cast<long long>(tp) * q.B + b, atn = static_cast<long long>(tn) * q.B + b;
      const float *pp = D.w + cell * q.stride + q.peep;
      in.p_i = pp[0]; in.p_f = pp[1]; in.p_o = pp[2];
      const float *g4 = (KIND == 1 ? D.gates_in : D.act) + at * 4 * C + cell;
#pragma unroll
      for (int k = 0; k < 4; ++k) in.g[k] = g4[k * C];
      if constexpr (KIND == 1) {
        in.cp = has_rec ? D.cstate[atp * C + cell] : 0.f;
        in.zs = D.zone_state == nullptr || D.zone_state[t * C + cell] != 0;
        in.zo = D.zone_output == nullptr || D.zone_output[t * C + cell] != 0;
        in.hp = !in.zo && has_rec ? D.values[atp * q.ldh + cell] : 0.f;
      } else {
        in.a = D.cact[at * C + cell];
        in.dh = D.deriv[at * q.ldh + cell];
        in.dni = in.dnf = in.dcn = in.fn = 0.f;
        if (has_rec) {
          const float *dn = D.dgates + atn * 4 * C + cell;
          in.dni = dn[C]; in.dnf = dn[2 * C];
          in.dcn = D.dcstate[atn * C + cell];
          in.fn = D.act[atn * 4 * C + 2 * C + cell];
        }
        in.cp = tp >= 0 && tp < q.T ? D.cstate[atp * C + cell] : 0.f;
      }
    };
    const bool early = q.RB == q.Rp && q.Rp * ncell <= LR_THREADS;
    if (early && tid < q.Rp * ncell && tid / ncell < nrow) load(tid / ncell, tid % ncell);
    if (has_rec && q.G > 1) {
      if (tid == 0 && !lr_wait(counter, static_cast<unsigned int>(q.G) * static_cast<unsigned int>(s), abort_word)) {
        s_ok = 0;
        atomicCAS(q.error_flag, 0, 411);
        atomicExch(abort_word, 1u);
      }
      __syncthreads();
      if (!s_ok) break;
    }
    const float *src = ex[(s & 1) ^ 1];
    float *dst = ex[s & 1];
    for (int rb = 0; rb < q.Rp; rb += q.RB) {
      const int rows_here = min(q.RB, q.Rp - rb);
      if (has_rec) {
        float acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int o = 0; o < 4; ++o) acc[r][o] = 0.f;
        const bool direct = q.G == 1;
        const int chunks = direct ? 1 : (q.K + q.KC - 1) / q.KC;
        const int buffers = chunks > 1 ? 2 : 1;
        const int groups4 = rows_here / 4;
        auto fetch = [&](int ch) {
          const int k0 = ch * q.KC, n = min(q.KC, q.K - k0) * groups4;
          float *to = in_s + (ch % buffers) * q.KC * q.RB;
          for (int i = tid; i < n; i += LR_THREADS) {
            const int k = i / groups4, r = (i - k * groups4) * 4;
            lr_copy16(to + k * q.RB + r, src + static_cast<size_t>(k0 + k) * q.Rp + rb + r);
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (!direct) fetch(0);
        for (int ch = 0; ch < chunks; ++ch) {
          int k0 = 0, n = q.K, pitch = q.Rp;
          const float *x = src + rb;
          if (!direct) {
            if (ch + 1 < chunks) {
              fetch(ch + 1);
              asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
              asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            k0 = ch * q.KC;
            n = min(q.KC, q.K - k0);
            x = in_s + (ch % buffers) * q.KC * q.RB;
            pitch = q.RB;
          }
          if (has_task && tile_r * 4 < rows_here) {
            const float *wp = w_s + static_cast<size_t>(k0) * q.NOp + col;
            const float *xp = x + tile_r * 4;
            const int step = 4 * q.KW;
#pragma unroll 4
            for (int k = kw * 4 + ks; k < n; k += step) {
              const float4 wv = *reinterpret_cast<const float4 *>(wp + k * q.NOp);
              const float4 xv = *reinterpret_cast<const float4 *>(xp + k * pitch);
              const float wo[4] = {wv.x, wv.y, wv.z, wv.w}, xr[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
              for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int o = 0; o < 4; ++o) acc[r][o] = fmaf(xr[r], wo[o], acc[r][o]);
            }
          }
          if (!direct && ch + 1 < chunks) __syncthreads();   // the buffer is refilled by the next but one fetch
        }
        // the four K slices of a warp: lane slice ks keeps row ks
        float half[2][4], mine[4];
        const bool up = (ks & 2) != 0, odd = (ks & 1) != 0;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int o = 0; o < 4; ++o) {
            const float keep = up ? acc[2 + r][o] : acc[r][o], give = up ? acc[r][o] : acc[2 + r][o];
            half[r][o] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
          }
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const float keep = odd ? half[1][o] : half[0][o], give = odd ? half[0][o] : half[1][o];
          mine[o] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
        }
        if (has_task && col_live && tile_r * 4 < rows_here)
          *reinterpret_cast<float4 *>(red_s + (static_cast<size_t>(kw) * q.RB + tile_r * 4 + ks) * q.NOp + col) = make_float4(mine[0], mine[1], mine[2], mine[3]);
        __syncthreads();
      }
      // one thread per (row, cell)
      for (int u = tid; u < rows_here * ncell; u += LR_THREADS) {
        const int rl = u / ncell, c = u - rl * ncell, rg = rb + rl;
        if (rg >= nrow) continue;   // padding of the row count
        if (!early) load(rg, c);
        const long long cell = cell0 + c, at = static_cast<long long>(t) * q.B + row0 + rg;
        if constexpr (KIND == 1) {
          float r4[4] = {0.f, 0.f, 0.f, 0.f};
          if (has_rec) {
            for (int k = 0; k < q.KW; ++k) {
              const float4 v = *reinterpret_cast<const float4 *>(red_s + (static_cast<size_t>(k) * q.RB + rl) * q.NOp + 4 * c);
              r4[0] += v.x; r4[1] += v.y; r4[2] += v.z; r4[3] += v.w;
            }
          }
          const float z = tanh_cell(in.g[0] + r4[0]);
          const float ig = sigmoid_cell(in.g[1] + (has_rec ? r4[1] + in.p_i * in.cp : 0.f));
          float fg = 0.f, cs = z * ig;
          if (has_rec) {
            fg = sigmoid_cell(in.g[2] + r4[2] + in.p_f * in.cp);
            cs += fg * in.cp;
          }
          if (!in.zs) cs = in.cp;
          const float a = tanh_cell(cs);
          const float og = sigmoid_cell(in.g[3] + r4[3] + in.p_o * cs);
          float h = a * og;
          if (!in.zo) h = in.hp;
          dst[cell * q.Rp + rg] = h;
          float *act = D.act + at * 4 * C + cell;
          act[0] = z; act[C] = ig; act[2 * C] = fg; act[3 * C] = og;
          D.cstate[at * C + cell] = cs;
          D.cact[at * C + cell] = a;
          D.values[at * q.ldh + cell] = h;
        } else {
          float dh = in.dh;
          if (has_rec) {
            float rec = 0.f;
            for (int k = 0; k < q.KW; ++k) rec += red_s[(static_cast<size_t>(k) * q.RB + rl) * q.NOp + c];
            dh += rec;
            D.deriv[at * q.ldh + cell] = dh;
          }
          const float z = in.g[0], ig = in.g[1], fg = in.g[2], og = in.g[3];
          const float d_o = og * (1.f - og) * (dh * in.a);
          float dc = dh * og * (1.f - in.a * in.a);
          dc += in.p_o * d_o;
          if (has_rec) {
            dc += in.p_i * in.dni;
            dc += in.p_f * in.dnf;
            dc += in.dcn * in.fn;
          }
          const float dz = dc * ig * (1.f - z * z);
          const float di = (dc * z) * (ig * (1.f - ig));
          const float df = tp >= 0 && tp < q.T ? (dc * in.cp) * (fg * (1.f - fg)) : 0.f;
          float *e = dst + cell * q.Rp + rg;
          const size_t gate_step = static_cast<size_t>(q.C) * q.Rp;
          e[0] = dz; e[gate_step] = di; e[2 * gate_step] = df; e[3 * gate_step] = d_o;
          float *dg = D.dgates + at * 4 * C + cell;
          dg[0] = dz; dg[C] = di; dg[2 * C] = df; dg[3 * C] = d_o;
          D.dcstate[at * C + cell] = dc;
        }
      }
      __syncthreads();   // red_s and (G = 1) the exchange buffer are complete / free again
    }
    if (q.G > 1 && tid == 0) lr_add_release(counter);
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
};

// shape of one kind for G CTAs per group; false when it does not fit.  clocks: estimate of a step
static bool resident_shape(int kind, long long B, long long C, int dirs, int sms, int G, ResidentArgs *q, size_t *smem, double *clocks) {
  const int cpc = static_cast<int>((C + G - 1) / G);
  if (static_cast<int>((C + cpc - 1) / cpc) != G) return false;
  const int max_groups = sms / (dirs * G);
  if (max_groups < 1) return false;
  q->G = G;
  q->cpc = cpc;
  q->C = static_cast<int>(C); q->B = static_cast<int>(B);
  q->R = static_cast<int>((B + max_groups - 1) / max_groups);
  q->Rp = (q->R + 3) / 4 * 4;
  q->groups = static_cast<int>((B + q->R - 1) / q->R);
  q->K = static_cast<int>(kind == 1 ? C : 4 * C);
  q->NOp = kind == 1 ? 4 * cpc : (cpc + 3) / 4 * 4;
  const int tiles_c = (q->NOp / 4 + 7) / 8;
  if (tiles_c > LR_WARPS) return false;
  q->RB = std::min(q->Rp, 4 * (LR_WARPS / tiles_c));
  const int tasks = tiles_c * (q->RB / 4);
  q->KW = LR_WARPS / tasks;
  // The whole exchange data of a pass where it fits: every chunk more is another trip to L2 within the step (1024 cells,
  // 16 rows: four chunks of 20 KB 11.3 us per step, one of 64 KB 9.7).
  const long long room = LR_SMEM_MAX / static_cast<long long>(sizeof(float)) - static_cast<long long>(q->K) * q->NOp - LR_RED_FLOATS;
  if (G == 1) {
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
  *smem = (static_cast<size_t>(q->K) * q->NOp + static_cast<size_t>(q->in_floats) + LR_RED_FLOATS) * sizeof(float);
  const double passes = static_cast<double>((q->Rp + q->RB - 1) / q->RB);
  const double reads = passes * tasks * (q->K / 4.0) * 5.0;                        // shared-memory wavefronts
  const double issue = passes * (q->K / (4.0 * q->KW)) * 20.0;                     // one warp's share, instruction by instruction
  const double exchange = G == 1 ? 0.0 : 3000.0 + 6.0 * G + q->K * static_cast<double>(q->Rp) * 4.0 / 40.0;
  const double chunks = (q->K + q->KC - 1) / q->KC;
  *clocks = std::max(reads, issue) + exchange + 900.0 * passes + 1000.0 * passes * (chunks - 1.0) + 300.0;
  return true;
}

// Which walk a pass takes.  The three are measured per time step and direction (us; weights loaded, T = 72 against T = 8):
//                     forward                            backward
//   cells x rows      resident  tensor  launches         resident  tensor  launches
//   128 x 32             3.2      6.5                       3.6      6.7
//   256 x 256            8.7     10.5                       9.8     12.9
//   301 x 512           31.8               27.7            31.7               32.3
//   512 x 32             5.9      8.9                       8.9     10.6
//   512 x 64             8.7      9.5                      15.3     11.7
//   512 x 128           14.4     11.4                      28.8     15.4
//   601 x 128           29.8               24.0            45.1               25.0
//   768 x 16             7.5     10.3                      12.5     12.2
//   768 x 32            11.9     10.5                      23.3     13.1
//   1001 x 4             5.0               20.3             9.1               21.7
//   1001 x 32           19.9               24.6            54.6               34.6
//   1024 x 4             4.9     11.7                       9.3     14.9
//   1024 x 16            9.5     11.7                      28.0     14.6
//   1024 x 32           16.4     11.8                      53.4     15.4
//   1024 x 256         113.8     14.7                     414.6     20.8
// Backward K is four times as long and only a quarter as wide, so the two passes cross at different sizes and are chosen by
// themselves (all walks leave the same arrays).  The estimates below are within 20 % of these times; resident_shape counts
// wavefronts and instructions and comes out 1.6 (forward) and 1.45 times (backward) below the clock.
static double resident_walk_us(int kind, double clocks) { return (kind == 1 ? 1.6 : 1.45) * clocks / 1900.0; }
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
  // best shape of either pass by itself, and of both with the same groups (where both are taken: the estimates of neighbouring
  // shapes are closer together than they are to the clock)
  LstmResident best, both;
  double best_clocks[2] = {1e30, 1e30}, sum_clocks = 1e30;
  for (int G = 1; G * P->dirs <= sms; ++G) {
    LstmResident r;
    double c[2] = {1e30, 1e30};
    const bool fits[2] = {resident_shape(1, net->B, P->C, P->dirs, sms, G, &r.f, &r.smem_f, &c[0]), resident_shape(2, net->B, P->C, P->dirs, sms, G, &r.b, &r.smem_b, &c[1])};
    if (fits[0] && c[0] < best_clocks[0]) { best_clocks[0] = c[0]; best.f = r.f; best.smem_f = r.smem_f; }
    if (fits[1] && c[1] < best_clocks[1]) { best_clocks[1] = c[1]; best.b = r.b; best.smem_b = r.smem_b; }
    if (fits[0] && fits[1] && c[0] + c[1] < sum_clocks) { sum_clocks = c[0] + c[1]; both = r; }
  }
  for (int k = 0; k < 2; ++k)
    P->resident_pass[k] = best_clocks[k] < 1e29 && resident_walk_us(k + 1, best_clocks[k]) < other_walk_us(P, k + 1, net->B) * P->dirs;
  if (P->resident_pass[0] && P->resident_pass[1] && sum_clocks < 1e29) best = both;
  if (!P->resident_pass[0] && !P->resident_pass[1]) return MYEA_OK;
  for (auto kernel : {lstm_resident_kernel<1>, lstm_resident_kernel<2>})
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LR_SMEM_MAX) != cudaSuccess) {
      cudaGetLastError();
      P->resident_pass[0] = P->resident_pass[1] = false;
      return MYEA_OK;
    }
  LstmResident *r = new LstmResident(best);
  P->resident = r;
  // (a pass that is not taken here has groups, K and Rp of its best shape or of none: both only size the buffers)
  const int counters = P->dirs * std::max(r->f.groups, r->b.groups);
  void *p = nullptr;
  const size_t ex_floats = 2 * static_cast<size_t>(P->dirs) * std::max(static_cast<size_t>(r->f.groups) * r->f.K * r->f.Rp, static_cast<size_t>(r->b.groups) * r->b.K * r->b.Rp);
  if (cudaMalloc(&p, ex_floats * sizeof(float)) != cudaSuccess) { net->ctx.error = "cudaMalloc failed (LSTM exchange buffer)"; return MYEA_E_CUDA; }
  net->allocations.push_back(p);
  r->ex = static_cast<float *>(p);
  if (cudaMemsetAsync(p, 0, ex_floats * sizeof(float), net->ctx.stream) != cudaSuccess) return MYEA_E_CUDA;  // rows that pad a group stay zero
  if (cudaMalloc(&p, (counters + 1) * sizeof(unsigned int)) != cudaSuccess) { net->ctx.error = "cudaMalloc failed (LSTM step counters)"; return MYEA_E_CUDA; }
  net->allocations.push_back(p);
  r->sync = static_cast<unsigned int *>(p);
  return MYEA_OK;
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
  if (q.G > 1 && cudaMemsetAsync(q.sync, 0, (q.sync_count + 1) * sizeof(unsigned int), ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(P->dirs * q.groups * q.G));
  cfg.blockDim = dim3(LR_THREADS);
  cfg.dynamicSmemBytes = kind == 1 ? r->smem_f : r->smem_b;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ctx.begin(TC_RECURRENT);
  const cudaError_t err = kind == 1 ? cudaLaunchKernelEx(&cfg, lstm_resident_kernel<1>, q) : cudaLaunchKernelEx(&cfg, lstm_resident_kernel<2>, q);
  ctx.end(TC_RECURRENT);
  ctx.gemm_flops += P->dirs * 2.0 * q.B * 4.0 * q.C * q.C * (q.T - 1);
  return err == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

}  // namespace myea
