// LSTM layer with peephole connections: forward pass, back-propagation through time, derivative-weight accumulation.
//
// Reference routines (Source_Files/Neural_Network/): forward Forward_Pass__LSTM__Gates_CIFO / __Gates_CIF_AF_State
// (and its Zoneout twin) / __States_AF / __Output (Neural_Network__Recurrent_Forward_Pass__OpenMP.cpp:859-1582), BPTT
// Backward_Pass__LSTM_Derivative__Output / __Cell_State_AF / __Gates_CIF_AF_State
// (Neural_Network__Recurrent_Backward_Pass__OpenMP.cpp:1130-1604), error to the previous layer Backward_Pass__LSTM (:1024-1120),
// Recurrent__Update_Derivative_Weight__LSTM + bias (Neural_Network__Recurrent_Update_Derivative_Weight__OpenMP.cpp:492-776).
//
// One cell per block (what every shipped configuration uses; blocks of several cells: lstm_blocks.cu).  Per step, with prev = the step before in the layer's direction:
//   z = tanh(Wz x + Rz h_prev + bz)          i = sig(Wi x + Ri h_prev + bi + pi*c_prev)
//   f = sig(Wf x + Rf h_prev + bf + pf*c_prev)   c = z*i + f*c_prev        (first step: no recurrent terms, no f)
//   o = sig(Wo x + Ro h_prev + bo + po*c)    h = tanh(c)*o
// Zoneout (forward only, as in the reference): where the state mask is false c = c_prev (0 at the first step), where
// the output mask is false h = h_prev (0 at the first step); the backward pass ignores the masks.
//
// Mapping to the GPU: the four gate matrices stay in the reference's interleaved per-block parameter layout.  The input
// projection of all T steps is ONE contraction [T*B, in] x [in, 4C] and the weight derivatives are contractions over K = T*B, for
// small products straight from the blocks (one launch for all gates), for large ones from operand panels (half_panels.cuh) that
// are split out of them.  The recurrent part is serial: one launch walks all steps of a layer where the weights fit shared
// memory (lstm_resident.cu) or the tiles of a step fit the chip (lstm_persistent.cu); else a [B, C] x [C, 4C] contraction and a
// fused cell kernel (gate nonlinearities, peepholes, cell-state recurrence, zoneout select) per step, and on the way back a
// [B, 4C] x [4C, C] contraction accumulated into the output error and a fused cell-backward kernel.  Bias and peephole
// derivatives are column reductions.
#include "half_panels.cuh"
#include "lstm.cuh"
#include "panel_math.cuh"

#include <algorithm>

namespace myea {

// offsets of the gate matrices inside one block of the parameter buffer (Prepare__Connections__LSTM)
struct BlockOffsets {
  long long z_in, z_rec, in[3], rec[3], peep;  // in/rec: input, forget, output gate
};
static BlockOffsets block_offsets(long long n_in, long long C) {
  BlockOffsets o;
  o.z_in = 0;
  o.z_rec = n_in;
  o.in[0] = n_in + C; o.in[1] = 2 * n_in + C; o.in[2] = 3 * n_in + C;
  o.rec[0] = 4 * n_in + C; o.rec[1] = 4 * n_in + 2 * C; o.rec[2] = 4 * n_in + 3 * C;
  o.peep = 4 * n_in + 4 * C;
  return o;
}

// ---------------------------------------------------------------------------------------------------------
// fused cell kernels
// ---------------------------------------------------------------------------------------------------------

struct CellFwd {
  const float *gates_in;  // rows of step t: [B, 4C]
  const float *s_rec;     // [B, 4C] or null at the first step
  const float *c_prev;    // [B, C] or null
  const float *h_prev;    // [B, ldh] or null
  const float *peep;      // parameter pointer of block 0's p_i; block c at + c*stride, p_f +1, p_o +2
  long long stride;
  float *act, *cstate, *cact, *h;  // rows of step t
  long long ldh;
  const uint8_t *zone_state, *zone_output;  // [C] of step t, or null
  long long B, C;
};

__global__ void __launch_bounds__(256) lstm_cell_forward_kernel(const CellFwd p) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long total = p.B * p.C;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long b = i / p.C, c = i - b * p.C;
    const float *gi = p.gates_in + b * 4 * p.C;
    const bool first = p.s_rec == nullptr;
    const float *sr = first ? nullptr : p.s_rec + b * 4 * p.C;
    const float pi = p.peep[c * p.stride], pf = p.peep[c * p.stride + 1], po = p.peep[c * p.stride + 2];
    const float cp = first ? 0.f : p.c_prev[b * p.C + c];
    const float sz = gi[c] + (first ? 0.f : sr[c]);
    const float si = gi[p.C + c] + (first ? 0.f : sr[p.C + c] + pi * cp);
    const float z = tanh_cell(sz);
    const float ig = sigmoid_cell(si);
    float fg = 0.f;
    float cs = z * ig;
    if (!first) {
      fg = sigmoid_cell(gi[2 * p.C + c] + sr[2 * p.C + c] + pf * cp);
      cs += fg * cp;
    }
    if (p.zone_state != nullptr && !p.zone_state[c]) cs = cp;  // cp is 0 at the first step
    const float a = tanh_cell(cs);
    const float og = sigmoid_cell(gi[3 * p.C + c] + (first ? 0.f : sr[3 * p.C + c]) + po * cs);
    float h = a * og;
    if (p.zone_output != nullptr && !p.zone_output[c]) h = first ? 0.f : p.h_prev[b * p.ldh + c];
    float *act = p.act + b * 4 * p.C;
    act[c] = z; act[p.C + c] = ig; act[2 * p.C + c] = fg; act[3 * p.C + c] = og;
    p.cstate[b * p.C + c] = cs;
    p.cact[b * p.C + c] = a;
    p.h[b * p.ldh + c] = h;
  }
}

struct CellBwd {
  const float *dh;        // [B, ldh] error on the outputs of step t (recurrent contribution already added)
  long long ldh;
  const float *act, *cact;     // step t
  const float *c_prev;         // cell state of the previous step in the layer's direction, null at the first step
  const float *act_next, *dgates_next, *dc_next;  // step after t in the layer's direction, null at the last step
  const float *peep;
  long long stride;
  float *dgates, *dcstate;     // step t
  long long B, C;
};

__global__ void __launch_bounds__(256) lstm_cell_backward_kernel(const CellBwd p) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long total = p.B * p.C;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long b = i / p.C, c = i - b * p.C;
    const float *act = p.act + b * 4 * p.C;
    const float z = act[c], ig = act[p.C + c], fg = act[2 * p.C + c], og = act[3 * p.C + c];
    const float a = p.cact[b * p.C + c];
    const float pi = p.peep[c * p.stride], pf = p.peep[c * p.stride + 1], po = p.peep[c * p.stride + 2];
    const float dh = p.dh[b * p.ldh + c];
    const float d_o = og * (1.f - og) * (dh * a);
    float dc = dh * og * (1.f - a * a);
    dc += po * d_o;
    if (p.dgates_next != nullptr) {
      const float *dn = p.dgates_next + b * 4 * p.C;
      dc += pi * dn[p.C + c];
      dc += pf * dn[2 * p.C + c];
      dc += p.dc_next[b * p.C + c] * p.act_next[b * 4 * p.C + 2 * p.C + c];
    }
    const float dz = dc * ig * (1.f - z * z);
    const float di = (dc * z) * (ig * (1.f - ig));
    const float df = p.c_prev != nullptr ? (dc * p.c_prev[b * p.C + c]) * (fg * (1.f - fg)) : 0.f;
    float *dg = p.dgates + b * 4 * p.C;
    dg[c] = dz; dg[p.C + c] = di; dg[2 * p.C + c] = df; dg[3 * p.C + c] = d_o;
    p.dcstate[b * p.C + c] = dc;
  }
}

// Bias and peephole derivatives: per cell c, over all rows r of dgates [R, 4C]
//   out0..3 = sum dz, di, df, do ; out4 = sum di[r]*c[r - shift], out5 = sum df[r]*c[r - shift] (rows whose partner
//   exists), out6 = sum do[r]*c[r].   partial[k][chunk][c].
__global__ void __launch_bounds__(256) lstm_bias_peephole_reduce_kernel(const float *__restrict__ dgates, const float *__restrict__ cstate,
                                                                        long long R, long long C, long long shift, int chunks,
                                                                        float *__restrict__ partial) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ float sh[7][8][33];
  const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const long long c = static_cast<long long>(blockIdx.x) * 32 + cl;
  const long long per = (R + chunks - 1) / chunks;
  const long long r0 = blockIdx.y * per, r1 = min(R, r0 + per);
  float acc[7] = {0, 0, 0, 0, 0, 0, 0};
  if (c < C) {
    for (long long r = r0 + rl; r < r1; r += 8) {
      const float *dg = dgates + r * 4 * C;
      const float dz = dg[c], di = dg[C + c], df = dg[2 * C + c], d_o = dg[3 * C + c];
      acc[0] += dz; acc[1] += di; acc[2] += df; acc[3] += d_o;
      const long long rp = r - shift;
      if (rp >= 0 && rp < R) {
        const float cs = cstate[rp * C + c];
        acc[4] = fmaf(di, cs, acc[4]);
        acc[5] = fmaf(df, cs, acc[5]);
      }
      acc[6] = fmaf(d_o, cstate[r * C + c], acc[6]);
    }
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) sh[k][rl][cl] = acc[k];
  __syncthreads();
  if (rl == 0 && c < C) {
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      float t = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) t += sh[k][r][cl];
      partial[(static_cast<long long>(k) * chunks + blockIdx.y) * C + c] = t;
    }
  }
}

// 32 cells per block, the chunks of a sum spread over 8 threads per cell
__global__ void __launch_bounds__(256) lstm_bias_peephole_finalize_kernel(const float *__restrict__ partial, int chunks, long long C, float *d_bias,
                                                                          float *d_peep, long long stride) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ float sh[7][8][33];
  const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const long long c = static_cast<long long>(blockIdx.x) * 32 + cl;
  float sum[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < C) {
#pragma unroll 4
    for (int ch = rl; ch < chunks; ch += 8) {
#pragma unroll
      for (int k = 0; k < 7; ++k) sum[k] += partial[(static_cast<long long>(k) * chunks + ch) * C + c];
    }
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) sh[k][rl][cl] = sum[k];
  __syncthreads();
  if (rl != 0 || c >= C) return;
  float t[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    t[k] = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) t[k] += sh[k][r][cl];
  }
  // atomics: with the reference's shifted bias base the output-gate slots alias the next layer's bias slots, which another
  // kernel of the same stream also accumulates into; stream order already serialises them, the atomics are belt and braces
  atomicAdd(&d_bias[c], t[0]);
  atomicAdd(&d_bias[C + c], t[1]);
  atomicAdd(&d_bias[2 * C + c], t[2]);
  atomicAdd(&d_bias[3 * C + c], t[3]);
  d_peep[c * stride] += t[4];
  d_peep[c * stride + 1] += t[5];
  d_peep[c * stride + 2] += t[6];
}

// peepholes p_i, p_f, p_o of every cell, gathered from the blocks of the parameter buffer into [3][C]
__global__ void lstm_gather_peepholes_kernel(const float *__restrict__ peep, long long stride, long long C, float *__restrict__ out) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (c >= C) return;
  out[c] = peep[c * stride];
  out[C + c] = peep[c * stride + 1];
  out[2 * C + c] = peep[c * stride + 2];
}

// the input (recurrent) weights of the four gates, [dirs][4C][width], out of the blocks (w0 / w1: first block of each
// direction; the cell input's row lies at off_z, the three gates' rows at off_gates, one after the other)
__global__ void __launch_bounds__(256) lstm_gather_weights_kernel(const float *__restrict__ w0, const float *__restrict__ w1, long long stride, long long off_z,
                                                                  long long off_gates, long long width, long long C, float *__restrict__ out) {
  grid_dependency_wait();
  // (no early release: in front of a walk by launches the first cells would set themselves up beside these blocks, the product of the
  // second step beside both, two of its CTAs to an SM, and every later step's like it: 701 cells, 200 rows 35 us per forward step, 52 then)
  const long long total = 4 * C * width;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / width, k = i - r * width, g = r / C, c = r - g * C;
    const long long at = c * stride + (g == 0 ? off_z : off_gates + (g - 1) * width) + k;
    out[i] = w0[at];
    if (w1 != nullptr) out[total + i] = w1[at];
  }
}

// ---------------------------------------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------------------------------------
template <typename T>
static int lalloc(myea_b200_net *net, T **p, size_t count) {
  void *q = nullptr;
  const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
  if (cudaMalloc(&q, bytes) != cudaSuccess) { net->ctx.error = "cudaMalloc failed (LSTM buffers)"; return MYEA_E_CUDA; }
  net->allocations.push_back(q);
  if (cudaMemsetAsync(q, 0, bytes, net->ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  *p = static_cast<T *>(q);
  return MYEA_OK;
}

#define LRC(expr) do { int rc__ = (expr); if (rc__ != MYEA_OK) return rc__; } while (0)

// memory for panels of a tensor that are made for one reading at a time
static size_t one_reading_floats(long long R, long long C) { return std::max(half_panel_floats(R, C, HALF_ROWS), half_panel_floats(R, C, HALF_COLS)); }

int lstm_create(myea_b200_net *net, LayerPlan &L) {
  const long long cpb = std::max<long long>(1, static_cast<long long>(L.desc.unit_parameters[1]));
  LstmPlan *P = new LstmPlan();
  L.lstm = P;
  P->dirs = L.desc.use_bidirectional ? 2 : 1;
  P->C = L.n_out / P->dirs;
  P->cpb = cpb;
  P->K = P->C / cpb;
  P->n_in = L.n_in;
  P->stride = static_cast<long long>(L.idx.block_stride);
  P->zoneout = L.desc.type_dropout == MYEA_DROPOUT_ZONEOUT;
  if (cpb != 1) return lstm_blocks_create(net, L, P);
  const long long rows = net->T * net->B, C = P->C;
  const bool tensor = net->ctx.gemm_engine == 0;
  const bool in_panels = tensor && !direct_gemm_suits(net->ctx, rows, 4 * C, L.n_in);
  const bool dw_panels = tensor && !direct_gemm_suits(net->ctx, 4 * C, std::max(L.n_in, C), rows);
  // biases: the reference stores first_bias_connection_index already shifted by the number of cells and then reads
  // [bz | bi | bf | bo] from it, so bo overlaps the next layer's bias slots.  Reproduced for the unidirectional layer;
  // the bidirectional layer (no usable reference) uses its true, unshifted block, one [bz|bi|bf|bo] run per direction.
  const long long fb = static_cast<long long>(L.idx.first_bias_connection_index);
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    D.w_base = static_cast<long long>(L.idx.first_connection_index) + d * C * P->stride;
    D.b_base = P->dirs == 1 ? fb : (fb - 2 * C) + d * 4 * C;
    if (D.b_base + 4 * C > static_cast<long long>(net->total_parameters)) {
      net->ctx.error = "LSTM output-gate bias would run past the parameter buffer (the next layer must be at least as wide as the LSTM layer)";
      return MYEA_E_INVALID;
    }
    // the input projections are dead after the forward walk, the gate errors' panels are made after the backward walk: one
    // buffer for both (of 268 MB at 1024 cells, 64 steps and 256 rows; mapping and clearing memory is most of what a handle costs)
    LRC(lalloc(net, &D.gates_in, in_panels || dw_panels ? std::max(static_cast<size_t>(rows * 4 * C), one_reading_floats(rows, 4 * C)) : static_cast<size_t>(rows * 4 * C)));
    if (in_panels || dw_panels) P->dg_all_mem[d] = D.gates_in;
    LRC(lalloc(net, &D.act, rows * 4 * C));
    LRC(lalloc(net, &D.cstate, rows * C));
    LRC(lalloc(net, &D.cact, rows * C));
    LRC(lalloc(net, &D.dgates, rows * 4 * C));
    LRC(lalloc(net, &D.dcstate, rows * C));
    if (P->zoneout) {
      LRC(lalloc(net, &D.zone_state, net->T * C));
      LRC(lalloc(net, &D.zone_output, net->T * C));
      cudaMemsetAsync(D.zone_state, 1, net->T * C, net->ctx.stream);
      cudaMemsetAsync(D.zone_output, 1, net->T * C, net->ctx.stream);
    }
  }
  LRC(lalloc(net, &L.values, rows * L.n_out));
  LRC(lalloc(net, &L.deriv, rows * L.n_out));
  L.errors = L.deriv;
  LRC(lalloc(net, &P->partial, static_cast<size_t>(7) * net->reduce_chunks * C));
  P->G = (C + 15) / 16 * 64;
  size_t need = static_cast<size_t>(P->dirs) * 4 * C * std::max<long long>(L.n_in, C);  // gathered weights
  LRC(lstm_persistent_plan(net, L));
  LRC(lstm_resident_plan(net, L));
  const bool walks[2] = {!P->resident_pass[0], !P->resident_pass[1]};   // passes that read the weights from what is laid out here
  const int w_readings = (walks[0] ? HALF_ROWS : 0) | (walks[1] ? HALF_COLS : 0);
  if (tensor && w_readings != 0 && lstm_persistent_ready(P)) {
    LRC(lalloc(net, &P->peep_compact, static_cast<size_t>(P->dirs) * 3 * C));
    const long long a_rows = (net->B + 127) / 128 * 128;
    float *mem = nullptr;
    if (walks[0]) {
      LRC(lalloc(net, &mem, half_panel_floats(2 * a_rows, C, HALF_ROWS)));       // zero: rows past the batch stay zero for ever
      P->h_pan = half_panels_at(mem, 2 * a_rows, C, HALF_ROWS);
    }
    if (walks[1]) {
      LRC(lalloc(net, &mem, half_panel_floats(2 * a_rows, P->G, HALF_ROWS)));
      P->dg_pan = half_panels_at(mem, 2 * a_rows, P->G, HALF_ROWS);
      LRC(lalloc(net, &P->dg_scale, static_cast<size_t>(2 * a_rows * (P->G / 64))));
    }
    LRC(lalloc(net, &P->w_rec_max, static_cast<size_t>(P->G + C)));
    for (int d = 0; d < P->dirs; ++d) {
      LRC(lalloc(net, &P->w_rec_mem[d], half_panel_floats(P->G, C, w_readings)));
      P->w_rec[d] = half_panels_at(P->w_rec_mem[d], P->G, C, w_readings);
      LRC(lalloc(net, &P->w_rec_scale[d], static_cast<size_t>(P->G + C)));
    }
  } else if (w_readings != 0) {
    if (walks[0]) LRC(lalloc(net, &P->s_rec, net->B * 4 * C));
    if (tensor && !direct_gemm_suits(net->ctx, net->B, 4 * C, C)) {
      for (int d = 0; d < P->dirs; ++d) {
        LRC(lalloc(net, &P->w_rec_mem[d], half_panel_floats(4 * C, C, w_readings)));
        P->w_rec[d] = half_panels_at(P->w_rec_mem[d], 4 * C, C, w_readings);
      }
      LRC(lalloc(net, &P->step_mem, half_panel_floats(net->B, 4 * C, HALF_ROWS)));
    } else {
      for (int d = 0; d < P->dirs; ++d) LRC(lalloc(net, &P->w_rec_mem[d], static_cast<size_t>(4 * C * C)));
    }
  }
  if (in_panels || dw_panels) LRC(lalloc(net, &P->x_mem, one_reading_floats(rows, L.n_in)));
  const int w_in_readings = L.input_layer > 0 ? HALF_BOTH : HALF_ROWS;   // (the network's inputs receive no error)
  for (int d = 0; d < P->dirs; ++d) {
    if (in_panels) {
      LRC(lalloc(net, &P->w_in_mem[d], half_panel_floats(4 * C, L.n_in, w_in_readings)));
      P->w_in[d] = half_panels_at(P->w_in_mem[d], 4 * C, L.n_in, w_in_readings);
    }
    if (dw_panels) LRC(lalloc(net, &P->h_shift_mem[d], half_panel_floats(rows, C, HALF_COLS)));
  }
  net->scratch.floats = std::max(net->scratch.floats, need + 256);
  return MYEA_OK;
}

void lstm_destroy(LayerPlan &L) {
  lstm_persistent_destroy(L.lstm);
  lstm_resident_destroy(L.lstm);
  delete L.lstm;
  L.lstm = nullptr;
}

float *lstm_output_errors(LayerPlan &L) { return L.deriv; }

int lstm_set_zoneout(myea_b200_net *net, LayerPlan &L, const uint8_t *state, const uint8_t *output, uint64_t count) {
  LstmPlan *P = L.lstm;
  if (P == nullptr || !P->zoneout || count != static_cast<uint64_t>(net->T * P->C * P->dirs)) {
    net->ctx.error = "layer has no zoneout masks of that size";
    return MYEA_E_INVALID;
  }
  // masks arrive as [T][dirs*C]
  for (int d = 0; d < P->dirs; ++d) {
    if (cudaMemcpy2DAsync(P->d[d].zone_state, P->C, state + d * P->C, P->dirs * P->C, P->C, net->T, cudaMemcpyHostToDevice, net->ctx.stream) != cudaSuccess ||
        cudaMemcpy2DAsync(P->d[d].zone_output, P->C, output + d * P->C, P->dirs * P->C, P->C, net->T, cudaMemcpyHostToDevice, net->ctx.stream) != cudaSuccess)
      return MYEA_E_CUDA;
  }
  return cudaStreamSynchronize(net->ctx.stream) == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// the per-direction zoneout arrays ([T][C] each) and probabilities of layer L, for the device-side mask generator
void lstm_zoneout_arrays(LayerPlan &L, int dir, uint8_t **state, uint8_t **output, long long *cells, int *dirs, float *p_state, float *p_output) {
  LstmPlan *P = L.lstm;
  *state = nullptr; *output = nullptr;
  if (P == nullptr || !P->zoneout || dir < 0 || dir >= P->dirs) return;
  *state = P->d[dir].zone_state;
  *output = P->d[dir].zone_output;
  *cells = P->C;
  *dirs = P->dirs;
  *p_state = L.desc.dropout_values[0];
  *p_output = L.desc.dropout_values[1];
}

static int cell_blocks(long long total) { return static_cast<int>(std::max<long long>(1, std::min<long long>((total + 255) / 256, 148 * 8))); }

// gate rows of the recurrent weights in the order (group of 16 cells, gate, cell): the tensor the persistent walk reads
struct GroupedGateRows {
  const float *w;
  long long stride, rec[4], C;
  bool vec;
  struct Cols {};
  __device__ __forceinline__ void columns(Cols &, long long, int) const {}
  __device__ __forceinline__ void row(const Cols &, long long r, long long c, int n, float (&v)[8]) const {
    const long long cell = (r >> 6) * 16 + (r & 15);
    const int g = static_cast<int>(r >> 4) & 3;
    if (cell < C) {
      ld8(v, w + cell * stride + rec[g] + c, n, vec);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
  }
  __device__ __forceinline__ void keep(long long, long long, int, const float (&)[8]) const {}
};
// Panels of the recurrent weights for the walk: a row (column) has ONE power of two for all of its K, so the walk, which finishes
// every sum once per step, multiplies by it once instead of stage by stage.  The largest magnitudes take a pass of their own
// (maxima: [G] of the rows, then [C] of the columns); both passes run when the weights have changed, 10 + 13 us for 1024 cells.
__global__ void __launch_bounds__(HP_THREADS, 2) weight_extents_kernel(const GroupedGateRows f, long long R, long long C, unsigned int *maxima) {
  grid_dependency_wait();
  grid_dependency_release();
  unsigned by, bx;
  half_block_of(C, blockIdx.x, by, bx);
  float v[HP_ROWS][8], m[HP_ROWS], mc[8];
  half_load_block(f, R, C, by, bx, v);
  half_row_maxima(v, m);
  half_column_maxima(v, mc);
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = by * static_cast<long long>(HP_BLOCK) + (threadIdx.x >> 4) + HP_THREADS / 16 * i;
    if ((threadIdx.x & 15) == 0 && r < R) atomicMax(maxima + r, __float_as_uint(m[i]));   // (magnitudes order like their bits)
  }
  if (threadIdx.x < 16) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long long c = bx * static_cast<long long>(HP_BLOCK) + threadIdx.x * 8 + j;
      if (c < C) atomicMax(maxima + R + c, __float_as_uint(mc[j]));
    }
  }
}
__global__ void __launch_bounds__(HP_THREADS, 2) weight_panels_kernel(const GroupedGateRows f, const HalfPanels p, const unsigned int *maxima, float *scale) {
  grid_dependency_wait();
  grid_dependency_release();
  unsigned by, bx;
  half_block_of(p.C, blockIdx.x, by, bx);
  float v[HP_ROWS][8], fc[8];
  half_load_block(f, p.R, p.C, by, bx, v);
  const long long c = bx * static_cast<long long>(HP_BLOCK) + (threadIdx.x & 15) * 8;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = c + j < p.C ? half_exponent(__uint_as_float(maxima[p.R + c + j])) : 0;
    fc[j] = pow2(-e);
    if (by == 0 && threadIdx.x < 16 && c + j < p.C) scale[p.R + c + j] = pow2(e);
  }
#pragma unroll
  for (int i = 0; i < HP_ROWS; ++i) {
    const long long r = by * static_cast<long long>(HP_BLOCK) + (threadIdx.x >> 4) + HP_THREADS / 16 * i;
    if (r >= p.R) continue;
    const int e = half_exponent(__uint_as_float(maxima[r]));
    if (bx == 0 && (threadIdx.x & 15) == 0) scale[r] = pow2(e);
    if (c >= p.pitch) continue;
    const float fr = pow2(-e);
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = v[i][j] * fr;
    if (p.rows.h0 != nullptr) half_store8(p, p.rows, r, c, s);
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = v[i][j] * fc[j];
    if (p.cols.h0 != nullptr) half_store8(p, p.cols, r, c, s);
  }
}
// rows of `src` shifted by `shift` rows, zeros where there is none
struct ShiftedRows {
  const float *src;
  long long pitch, shift, rows;
  bool vec;
  struct Cols {};
  __device__ __forceinline__ void columns(Cols &, long long, int) const {}
  __device__ __forceinline__ void row(const Cols &, long long r, long long c, int n, float (&v)[8]) const {
    const long long s = r - shift;
    if (s >= 0 && s < rows) {
      ld8(v, src + s * pitch + c, n, vec);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
  }
  __device__ __forceinline__ void keep(long long, long long, int, const float (&)[8]) const {}
};
static bool vec8(const float *p, long long a, long long b = 0) { return ((reinterpret_cast<uintptr_t>(p) & 15) == 0) && ((a | b) & 3) == 0; }

// ---------------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------------
static int prepare_input(myea_b200_net *net, LstmPlan *P, const float *input, long long rows, long long n_in, int reading) {
  if (P->x_src == input && P->x_reading == reading) return MYEA_OK;
  P->x = half_panels_at(P->x_mem, rows, n_in, reading);
  LRC(half_split(net->ctx, input, n_in, P->x));
  P->x_src = input;
  P->x_reading = reading;
  return MYEA_OK;
}

// the recurrent weights as the walks that do not keep them resident read them; made by the first of them after the parameters
// have changed
static int lay_out_recurrent_weights(myea_b200_net *net, LstmPlan *P, const BlockOffsets &off) {
  if (P->w_rec_fresh) return MYEA_OK;
  Context &ctx = net->ctx;
  const long long C = P->C, rec[4] = {off.z_rec, off.rec[0], off.rec[1], off.rec[2]};
  for (int d = 0; d < P->dirs; ++d) {
    const float *w = net->params + P->d[d].w_base;
    if (lstm_persistent_ready(P)) {
      ctx.begin(TC_RECURRENT);
      launch_dependent(ctx, lstm_gather_peepholes_kernel, dim3(static_cast<unsigned>((C + 255) / 256)), dim3(256), 0, w + off.peep, P->stride, C, P->peep_compact + static_cast<size_t>(d) * 3 * C);
      ctx.end(TC_RECURRENT);
      ctx.begin(TC_SPLIT);
      const GroupedGateRows src{w, P->stride, {rec[0], rec[1], rec[2], rec[3]}, C, vec8(w, P->stride, rec[0] | rec[1] | rec[2] | rec[3])};
      const dim3 grid(half_blocks(P->G, C)), block(HP_THREADS);
      if (cudaMemsetAsync(P->w_rec_max, 0, static_cast<size_t>(P->G + C) * sizeof(unsigned int), ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
      launch_dependent(ctx, weight_extents_kernel, grid, block, 0, src, P->G, C, P->w_rec_max);
      launch_dependent(ctx, weight_panels_kernel, grid, block, 0, src, P->w_rec[d], static_cast<const unsigned int *>(P->w_rec_max), P->w_rec_scale[d]);
      ctx.end(TC_SPLIT, 2);
    } else if (P->step_mem != nullptr) {
      RowSegments seg;
      seg.seg_rows = C;
      for (int g = 0; g < 4; ++g) seg.seg_off[g] = rec[g];
      LRC(half_split(ctx, w, P->stride, P->w_rec[d], &seg));
    } else {
      ctx.begin(TC_RECURRENT);
      launch_dependent(ctx, lstm_gather_weights_kernel, dim3(static_cast<unsigned>(std::min<long long>((4 * C * C + 255) / 256, 148 * 8))), dim3(256), 0, w, nullptr, P->stride, rec[0], rec[1], C, C,
                                                                                                                                   P->w_rec_mem[d]);
      ctx.end(TC_RECURRENT);
    }
  }
  P->w_rec_fresh = true;
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

int lstm_forward(myea_b200_net *net, LayerPlan &L, const float *input, long long n_in) {
  LstmPlan *P = L.lstm;
  if (P->cpb != 1) return lstm_blocks_forward(net, L, input, n_in);
  Context &ctx = net->ctx;
  const long long T = net->T, B = net->B, rows = T * B, C = P->C, ldh = L.n_out;
  const BlockOffsets off = block_offsets(n_in, C);
  P->x_src = nullptr;
  P->dg_all_reading[0] = P->dg_all_reading[1] = 0;
  // input projection of all steps: gates_in = x W_in^T + b, columns [z | i | f | o]
  if (P->w_in_mem[0] == nullptr) {  // the four gates (of both directions) in one launch, straight from the blocks
    DirectItem items[8];
    int n = 0;
    for (int d = 0; d < P->dirs; ++d)
      for (int g = 0; g < 4; ++g) {
        DirectItem &it = items[n++];
        it.A = Operand{input, rows, n_in, n_in, 1};
        it.B = Operand{net->params + P->d[d].w_base + (g == 0 ? off.z_in : off.in[g - 1]), C, n_in, P->stride, 1};
        it.epi.C = P->d[d].gates_in + g * C;
        it.epi.ldc = 4 * C;
        it.epi.bias = net->params + P->d[d].b_base + g * C;
      }
    if (ctx.gemm_engine == 0) {
      LRC(direct_gemm(ctx, items, n));
    } else {
      for (int i = 0; i < n; ++i) LRC(gemm_nt(ctx, items[i].A, items[i].B, items[i].epi, net->scratch));
    }
  } else {
    LRC(prepare_input(net, P, input, rows, n_in, HALF_ROWS));
    for (int d = 0; d < P->dirs; ++d) {
      if (!L.w_fresh) {
        RowSegments seg;
        seg.seg_rows = C;
        seg.seg_off[0] = off.z_in;
        for (int g = 0; g < 3; ++g) seg.seg_off[g + 1] = off.in[g];
        LRC(half_split(ctx, net->params + P->d[d].w_base, P->stride, P->w_in[d], &seg));
      }
      Epilogue e;
      e.C = P->d[d].gates_in;
      e.ldc = 4 * C;
      e.bias = net->params + P->d[d].b_base;
      LRC(half_gemm(ctx, half_rows(P->x), half_rows(P->w_in[d]), e));
    }
  }
  const bool zone = P->zoneout && net->training;
  if (!L.w_fresh) P->w_rec_fresh = false;
  L.w_fresh = true;   // (what is laid out from the weights stays until the parameters change)
  if (P->resident_pass[0]) {
    const long long rec[4] = {off.z_rec, off.rec[0], off.rec[1], off.rec[2]};
    return lstm_resident_run(net, L, 1, zone, rec, off.peep);
  }
  LRC(lay_out_recurrent_weights(net, P, off));
  if (lstm_persistent_ready(P)) {
    for (int d = 0; d < P->dirs; ++d) LRC(lstm_persistent_forward(net, L, d, zone));
    return MYEA_OK;
  }
  // the walk by launches: per step the recurrent product and the cell kernel
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    const float *w = net->params + D.w_base;
    for (long long s = 0; s < T; ++s) {
      const long long t = d == 0 ? s : T - 1 - s;
      const long long tp = d == 0 ? t - 1 : t + 1;
      CellFwd cf;
      cf.gates_in = D.gates_in + t * B * 4 * C;
      cf.s_rec = nullptr; cf.c_prev = nullptr; cf.h_prev = nullptr;
      if (s > 0) {
        const float *h_prev = L.values + tp * B * ldh + d * C;
        Epilogue er;
        er.C = P->s_rec;
        er.ldc = 4 * C;
        if (P->step_mem != nullptr) {
          const HalfPanels ph = half_panels_at(P->step_mem, B, C, HALF_ROWS);
          LRC(half_split(ctx, h_prev, ldh, ph));
          LRC(half_gemm(ctx, half_rows(ph), half_rows(P->w_rec[d]), er));
        } else {
          LRC(gemm_nt(ctx, Operand{h_prev, B, C, ldh, 1}, Operand{P->w_rec_mem[d], 4 * C, C, C, 1}, er, net->scratch));
        }
        cf.s_rec = P->s_rec;
        cf.c_prev = D.cstate + tp * B * C;
        cf.h_prev = h_prev;
      }
      cf.peep = w + off.peep;
      cf.stride = P->stride;
      cf.act = D.act + t * B * 4 * C;
      cf.cstate = D.cstate + t * B * C;
      cf.cact = D.cact + t * B * C;
      cf.h = L.values + t * B * ldh + d * C;
      cf.ldh = ldh;
      cf.zone_state = zone ? D.zone_state + t * C : nullptr;
      cf.zone_output = zone ? D.zone_output + t * C : nullptr;
      cf.B = B; cf.C = C;
      ctx.begin(TC_RECURRENT);
      launch_dependent(ctx, lstm_cell_forward_kernel, dim3(cell_blocks(B * C)), dim3(256), 0, cf);
      ctx.end(TC_RECURRENT);
    }
  }
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// ---------------------------------------------------------------------------------------------------------
// BPTT: L.deriv holds the error arriving on the layer's outputs from its consumers
// ---------------------------------------------------------------------------------------------------------
int lstm_backward(myea_b200_net *net, LayerPlan &L) {
  LstmPlan *P = L.lstm;
  if (P->cpb != 1) return lstm_blocks_backward(net, L);
  Context &ctx = net->ctx;
  const long long T = net->T, B = net->B, C = P->C, ldh = L.n_out, n_in = P->n_in;
  const BlockOffsets off = block_offsets(n_in, C);
  P->dg_all_reading[0] = P->dg_all_reading[1] = 0;
  if (P->resident_pass[1]) {
    const long long rec[4] = {off.z_rec, off.rec[0], off.rec[1], off.rec[2]};
    return lstm_resident_run(net, L, 2, false, rec, off.peep);
  }
  LRC(lay_out_recurrent_weights(net, P, off));
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    if (lstm_persistent_ready(P)) {
      LRC(lstm_persistent_backward(net, L, d));
      continue;
    }
    for (long long s = 0; s < T; ++s) {
      const long long t = d == 0 ? T - 1 - s : s;      // walk against the layer's direction
      const long long tn = d == 0 ? t + 1 : t - 1;     // the step after t in the layer's direction
      const long long tp = d == 0 ? t - 1 : t + 1;     // the step before t
      float *dh_t = L.deriv + t * B * ldh + d * C;
      if (s > 0) {  // error through time: the gate errors of the step after times the recurrent weights
        const float *dg = D.dgates + tn * B * 4 * C;
        Epilogue e;
        e.C = dh_t;
        e.ldc = ldh;
        e.accumulate = 1;
        if (P->step_mem != nullptr) {
          const HalfPanels pd = half_panels_at(P->step_mem, B, 4 * C, HALF_ROWS);
          LRC(half_split(ctx, dg, 4 * C, pd));
          LRC(half_gemm(ctx, half_rows(pd), half_cols(P->w_rec[d]), e));
        } else {
          LRC(gemm_nt(ctx, Operand{dg, B, 4 * C, 4 * C, 1}, Operand{P->w_rec_mem[d], C, 4 * C, 1, C}, e, net->scratch));
        }
      }
      CellBwd cb;
      cb.dh = dh_t;
      cb.ldh = ldh;
      cb.act = D.act + t * B * 4 * C;
      cb.cact = D.cact + t * B * C;
      cb.c_prev = (tp >= 0 && tp < T) ? D.cstate + tp * B * C : nullptr;
      cb.act_next = s > 0 ? D.act + tn * B * 4 * C : nullptr;
      cb.dgates_next = s > 0 ? D.dgates + tn * B * 4 * C : nullptr;
      cb.dc_next = s > 0 ? D.dcstate + tn * B * C : nullptr;
      cb.peep = net->params + D.w_base + off.peep;
      cb.stride = P->stride;
      cb.dgates = D.dgates + t * B * 4 * C;
      cb.dcstate = D.dcstate + t * B * C;
      cb.B = B; cb.C = C;
      ctx.begin(TC_RECURRENT);
      launch_dependent(ctx, lstm_cell_backward_kernel, dim3(cell_blocks(B * C)), dim3(256), 0, cb);
      ctx.end(TC_RECURRENT);
    }
  }
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// the gate errors of all steps as panels: read through their rows by the error to the layer below, through their columns by
// the weight derivatives.  One after the other in the same memory: both at once would double the largest buffer of a layer, and
// clearing it is most of what creating a handle costs; the second pass over the gate errors is 0.5 % of a step.
static int prepare_gate_errors(myea_b200_net *net, LstmPlan *P, int d, long long rows, int reading) {
  if (P->dg_all_reading[d] == reading) return MYEA_OK;
  P->dg_all[d] = half_panels_at(P->dg_all_mem[d], rows, 4 * P->C, reading);
  LRC(half_split(net->ctx, P->d[d].dgates, 4 * P->C, P->dg_all[d]));
  P->dg_all_reading[d] = reading;
  return MYEA_OK;
}

// error of the LSTM layer L propagated to the outputs of the layer feeding it: prev_deriv [T*B, n_in] = sum over
// directions of dgates [T*B, 4C] * W_in [4C, n_in].  `finish` (optional) carries the activation derivative of a fully
// connected layer below, applied by the epilogue of the last direction's contraction to the complete sum.
int lstm_backward_to_input(myea_b200_net *net, LayerPlan &L, float *prev_deriv, const LayerPlan &prev, const Epilogue *finish) {
  LstmPlan *P = L.lstm;
  if (P->cpb != 1) return lstm_blocks_backward_to_input(net, L, prev_deriv, prev, finish);
  Context &ctx = net->ctx;
  const long long rows = net->T * net->B, C = P->C, n_in = P->n_in;
  if (prev.n_out != n_in) return MYEA_E_INVALID;
  const BlockOffsets off = block_offsets(n_in, C);
  const bool gathered = P->w_in_mem[0] == nullptr;
  if (gathered) {  // the input weights gathered out of the blocks once (their four gate matrices are one K range then)
    ctx.begin(TC_RECURRENT);
    launch_dependent(ctx, lstm_gather_weights_kernel, dim3(static_cast<unsigned>(std::min<long long>((4 * C * n_in + 255) / 256, 148 * 8))), dim3(256), 0, 
        net->params + P->d[0].w_base, P->dirs > 1 ? net->params + P->d[1].w_base : nullptr, P->stride, off.z_in, off.in[0], n_in, C, net->scratch.base);
    ctx.end(TC_RECURRENT);
  }
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    Epilogue e;
    if (finish != nullptr && d == P->dirs - 1) e = *finish;
    e.C = prev_deriv;
    e.ldc = n_in;
    if (d > 0 && finish != nullptr) { e.addend = prev_deriv; e.ld_addend = n_in; }  // the addend enters before the derivative
    else e.accumulate = d > 0 ? 1 : 0;
    if (gathered) {
      const DirectItem it{Operand{D.dgates, rows, 4 * C, 4 * C, 1}, Operand{net->scratch.base + d * 4 * C * n_in, n_in, 4 * C, 1, n_in}, e, nullptr};
      if (ctx.gemm_engine == 0) LRC(direct_gemm(ctx, &it, 1));
      else LRC(gemm_nt(ctx, it.A, it.B, e, GemmScratch{}));
    } else {
      LRC(prepare_gate_errors(net, P, d, rows, HALF_ROWS));
      LRC(half_gemm(ctx, half_rows(P->dg_all[d]), half_cols(P->w_in[d]), e));
    }
  }
  return MYEA_OK;
}

// ---------------------------------------------------------------------------------------------------------
// derivative weights: dW_in,g += dg^T x ; dW_rec,g += dg(next step)^T h ; peepholes and biases by column reductions
// ---------------------------------------------------------------------------------------------------------
int lstm_update_derivative_weight(myea_b200_net *net, LayerPlan &L, const float *input, long long n_in) {
  LstmPlan *P = L.lstm;
  if (P->cpb != 1) return lstm_blocks_update_derivative_weight(net, L, input, n_in);
  Context &ctx = net->ctx;
  const long long T = net->T, B = net->B, rows = T * B, C = P->C, ldh = L.n_out;
  const BlockOffsets off = block_offsets(n_in, C);
  for (int d = 0; d < P->dirs; ++d) {
    LstmDir &D = P->d[d];
    float *gw = net->grads + D.w_base;
    const long long shift = d == 0 ? B : -B;   // rows of time step t against the outputs one step earlier in the direction
    if (P->h_shift_mem[0] == nullptr) {
      // gate by gate in one launch: the gate errors against the layer's input and against its output one step earlier
      DirectItem items[8];
      const long long K = (T - 1) * B;
      const float *dg0 = d == 0 ? D.dgates + B * 4 * C : D.dgates;
      const float *h0 = d == 0 ? L.values + d * C : L.values + B * ldh + d * C;
      int n = 0;
      for (int g = 0; g < 4; ++g) {
        DirectItem &it = items[n++];
        it.A = Operand{D.dgates + g * C, C, rows, 1, 4 * C};
        it.B = Operand{input, n_in, rows, 1, n_in};
        it.epi.C = gw + (g == 0 ? off.z_in : off.in[g - 1]);
        it.epi.ldc = P->stride;
        it.epi.accumulate = 1;
        if (T > 1) {
          DirectItem &r = items[n++];
          r.A = Operand{dg0 + g * C, C, K, 1, 4 * C};
          r.B = Operand{h0, C, K, 1, ldh};
          r.epi.C = gw + (g == 0 ? off.z_rec : off.rec[g - 1]);
          r.epi.ldc = P->stride;
          r.epi.accumulate = 1;
        }
      }
      if (ctx.gemm_engine == 0) {
        LRC(direct_gemm(ctx, items, n));
      } else {
        for (int i = 0; i < n; ++i) LRC(gemm_nt(ctx, items[i].A, items[i].B, items[i].epi, GemmScratch{}));
      }
    } else {
      // the four gates in one contraction: row g*C + c of the product lands in block c at gate g's offset
      LRC(prepare_input(net, P, input, rows, n_in, HALF_COLS));
      LRC(prepare_gate_errors(net, P, d, rows, HALF_COLS));
      Epilogue e;
      e.C = gw;
      e.ldc = P->stride;
      e.accumulate = 1;
      e.seg_rows = C;
      e.seg_off[0] = off.z_in;
      for (int g = 0; g < 3; ++g) e.seg_off[g + 1] = off.in[g];
      LRC(half_gemm(ctx, half_cols(P->dg_all[d]), half_cols(P->x), e));
      if (T > 1) {
        // recurrent weights over all rows too: the outputs shifted by one step, zeros at the direction's first step
        const HalfPanels hs = half_panels_at(P->h_shift_mem[d], rows, C, HALF_COLS);
        ctx.begin(TC_SPLIT);
        half_produce(ctx, ShiftedRows{L.values + d * C, ldh, shift, rows, vec8(L.values, ldh, C)}, hs);
        ctx.end(TC_SPLIT);
        e.seg_off[0] = off.z_rec;
        for (int g = 0; g < 3; ++g) e.seg_off[g + 1] = off.rec[g];
        LRC(half_gemm(ctx, half_cols(P->dg_all[d]), half_cols(hs), e));
      }
    }
    // biases and peepholes
    const int chunks = static_cast<int>(std::max<long long>(1, std::min<long long>(net->reduce_chunks, rows / 8)));
    ctx.begin(TC_RECURRENT);
    dim3 grid(static_cast<unsigned>((C + 31) / 32), chunks);
    launch_dependent(ctx, lstm_bias_peephole_reduce_kernel, grid, dim3(256), 0, D.dgates, D.cstate, rows, C, shift, chunks, P->partial);
    launch_dependent(ctx, lstm_bias_peephole_finalize_kernel, dim3(static_cast<unsigned>((C + 31) / 32)), dim3(256), 0, P->partial, chunks, C, net->grads + D.b_base,
                                                                                                    gw + off.peep, P->stride);
    ctx.end(TC_RECURRENT, 2);
  }
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// how far reciprocal_from_one is from the correctly rounded reciprocal over `count` floats from the bit pattern `first` on
__global__ void __launch_bounds__(256) reciprocal_check_kernel(unsigned int first, unsigned int count, unsigned long long *different, unsigned int *most) {
  unsigned long long n = 0;
  unsigned int worst = 0;
  for (unsigned int i = blockIdx.x * 256u + threadIdx.x; i < count; i += gridDim.x * 256u) {
    const float d = __uint_as_float(first + i);
    const int ulps = abs(__float_as_int(reciprocal_from_one(d)) - __float_as_int(__frcp_rn(d)));
    n += ulps != 0;
    worst = max(worst, static_cast<unsigned int>(ulps));
  }
  if (n != 0) atomicAdd(different, n);
  atomicMax(most, worst);
}

}  // namespace myea

// Diagnostic (not part of the training interface): over the floats with bit patterns first .. first + count - 1 (positive), how many
// reciprocals of the LSTM cells differ from the correctly rounded ones, and by how many units in the last place at most.
extern "C" int myea_b200_reciprocal_check(int device, uint32_t first, uint32_t count, uint64_t *different, uint32_t *most) {
  if (different == nullptr || most == nullptr || first > 0x7f800000u || count > 0x7f800000u - first) return MYEA_E_INVALID;
  if (cudaSetDevice(device) != cudaSuccess) return MYEA_E_CUDA;
  unsigned long long *out = nullptr;   // [0] count, [1] maximum
  if (cudaMalloc(&out, 2 * sizeof(*out)) != cudaSuccess) return MYEA_E_CUDA;
  unsigned long long got[2] = {0, 0};
  const bool ok = cudaMemset(out, 0, sizeof(got)) == cudaSuccess &&
                  (myea::reciprocal_check_kernel<<<148 * 8, 256>>>(first, count, out, reinterpret_cast<unsigned int *>(out + 1)), cudaGetLastError() == cudaSuccess) &&
                  cudaMemcpy(got, out, sizeof(got), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(out);
  *different = got[0];
  *most = static_cast<uint32_t>(got[1]);
  return ok ? MYEA_OK : MYEA_E_CUDA;
}
