// Plan of one LSTM layer on the device (lstm.cu) and the persistent step kernels that walk its time steps
// (lstm_persistent.cu).
#pragma once

#include "net.cuh"

namespace myea {

struct LstmDir {
  long long w_base = 0;   // first parameter of this direction's blocks
  long long b_base = 0;   // [bz (C) | bi (C) | bf (C) | bo (C)]
  float *gates_in = nullptr;  // [T*B, 4C] input projection + bias, columns [z | i | f | o]
  float *act = nullptr;       // [T*B, 4C] activated gates
  float *cstate = nullptr, *cact = nullptr;  // [T*B, C] cell state, tanh(cell state)
  float *dgates = nullptr;    // [T*B, 4C] error w.r.t. the gate summations
  float *dcstate = nullptr;   // [T*B, C]
  uint8_t *zone_state = nullptr, *zone_output = nullptr;  // [T, C], 1 = compute, 0 = keep the previous value
};

struct LstmPersistent;
struct LstmResident;
struct LstmPlan {
  int dirs = 1;
  long long C = 0, n_in = 0, stride = 0;
  bool zoneout = false;
  LstmDir d[2];
  float *s_rec = nullptr;      // [B, 4C] recurrent projection of the current step (walk by launches)
  float *partial = nullptr;    // [7][chunks][C]
  float *peep_compact = nullptr;  // [dirs][3][C]
  // Operand panels (half_panels.cuh) of contractions too large for the products straight from fp32.  x: layer input [T*B, in];
  // w_in: the four gates' input weights [4C, in]; dg_all: gate errors [T*B, 4C]; h_shift: the layer's outputs one step
  // earlier in the direction [T*B, C] (zeros at its first step).
  float *x_mem = nullptr, *w_in_mem[2] = {nullptr, nullptr}, *dg_all_mem[2] = {nullptr, nullptr}, *h_shift_mem[2] = {nullptr, nullptr};
  HalfPanels x, w_in[2], dg_all[2];
  // x and dg_all hold the panels of one reading at a time: through rows for the products on the way forward and back, through
  // columns for the weight derivatives behind them
  const float *x_src = nullptr;   // the array the x panels were made from in this step, and their reading
  int x_reading = 0;
  int dg_all_reading[2] = {0, 0};   // 0: not made in this step
  // Recurrent weights as panels: for the persistent walk [G, C] with the gate rows in the order (group of 16 cells, gate,
  // cell), G = 64 * ceil(C / 16), and one power of two for ALL of K (w_rec_scale: [G] of the rows, [C] of the columns; the walk
  // multiplies by it once per step); for the walk by launches [4C, C] gate after gate, or (small products) gathered in fp32.
  long long G = 0;
  float *w_rec_mem[2] = {nullptr, nullptr};
  HalfPanels w_rec[2];
  float *w_rec_scale[2] = {nullptr, nullptr};
  unsigned int *w_rec_max = nullptr;   // [G + C] largest magnitudes on the way to the scales
  // Ping-pong operand panels of the persistent walk, both buffers in one tensor of 2 * a_rows rows (a_rows: the batch rounded up to
  // 128): h [.., C] with a fixed exponent, gate errors [.., G] with powers of two [2][rows / 128][G / 64][128 rows]
  HalfPanels h_pan, dg_pan;
  uint16_t *dg_scale = nullptr;
  float *step_mem = nullptr;   // walk by launches: panels of one step's operand
  LstmPersistent *persist = nullptr;
  LstmResident *resident = nullptr;  // the walk with resident weights (lstm_resident.cu)
  bool resident_pass[2] = {false, false};   // whether the forward / backward pass takes it
  bool w_rec_fresh = false;                 // the recurrent weights as the other walks read them match the parameters
  // blocks of several cells (lstm_blocks.cu): K blocks of cpb cells per direction, gate rows of G = C + 3K columns
  // [z (C) | i (K) | f (K) | o (K)], weights gathered into dense matrices for the pass and their derivatives scattered back
  long long K = 0, cpb = 1;
  float *blk_w_in = nullptr, *blk_w_rec = nullptr, *blk_peep = nullptr;       // [G, in], [G, C], [3][C]
  float *blk_dw_in = nullptr, *blk_dw_rec = nullptr, *blk_dpeep = nullptr;
  float *blk_products = nullptr;                                               // [T*B, 3C]
};

int lstm_blocks_create(myea_b200_net *net, LayerPlan &L, LstmPlan *P);
int lstm_blocks_forward(myea_b200_net *net, LayerPlan &L, const float *input, long long n_in);
int lstm_blocks_backward(myea_b200_net *net, LayerPlan &L);
int lstm_blocks_backward_to_input(myea_b200_net *net, LayerPlan &L, float *prev_deriv, const LayerPlan &prev, const Epilogue *finish);
int lstm_blocks_update_derivative_weight(myea_b200_net *net, LayerPlan &L, const float *input, long long n_in);


// One launch that walks ALL time steps of one layer and direction (lstm_persistent.cu): the recurrent
// contraction of every step on the tensor cores, the cell arithmetic in its epilogue, the step's results written as the
// next step's operand panels, and a bounded grid-wide barrier between steps.
//   forward: steps s = 0 .. T-1 of direction `dir` (step s reads the h panels of buffer (s - 1) & 1)
//   backward: steps s = 0 .. T-1 of the walk against the direction (step s reads the gate-error panels of (s - 1) & 1)
// lstm_persistent_plan decides at creation whether the layer's shapes fit (every tile resident at once); the step
// functions return MYEA_E_UNSUPPORTED when they do not apply and the caller takes the per-step path.
int lstm_persistent_plan(myea_b200_net *net, LayerPlan &L);
void lstm_persistent_destroy(LstmPlan *P);
bool lstm_persistent_ready(const LstmPlan *P);
int lstm_persistent_forward(myea_b200_net *net, LayerPlan &L, int dir, bool zoneout);
int lstm_persistent_backward(myea_b200_net *net, LayerPlan &L, int dir);

// The walk for small batches and narrow or odd layers: all time steps (and both directions) in one launch, recurrent weights
// in shared memory, read from the parameter buffer itself.  lstm_resident_plan decides which passes take it.
int lstm_resident_plan(myea_b200_net *net, LayerPlan &L);
void lstm_resident_destroy(LstmPlan *P);
bool lstm_resident_stall(LstmPlan *P, int step, long long cycles);
int lstm_resident_run(myea_b200_net *net, LayerPlan &L, int kind, bool zoneout, const long long rec[4], long long peep);

}  // namespace myea
