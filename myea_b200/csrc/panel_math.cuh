// The arithmetic of one LSTM cell step for 8 consecutive cells of one batch row, and how its results leave as operand panels
// of the next step (lstm_persistent.cu); the activation functions as lstm.cu has them.
#pragma once

#include "common.cuh"
#include "half_panels.cuh"

namespace myea {

__device__ __forceinline__ void load8(float (&d)[8], const float *p) {
  const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}
__device__ __forceinline__ void store8(float *p, const float (&d)[8]) {
  *reinterpret_cast<float4 *>(p) = make_float4(d[0], d[1], d[2], d[3]);
  *reinterpret_cast<float4 *>(p + 4) = make_float4(d[4], d[5], d[6], d[7]);
}
// One time step of an LSTM layer as the cell arithmetic sees it: the arrays of step t, of the step before / after it in
// the layer's direction, and where the results also leave as operand panels of the next step's contraction.
struct LstmStep {
  long long C = 0, ldh = 0, kp = 0;
  const float *peep = nullptr;  // compact peepholes [3][C]: p_i, p_f, p_o
  uint16_t *p_h0 = nullptr, *p_h1 = nullptr;  // operand panels written for the next step (pitch kp), or null
  // forward (rows of step t unless said otherwise)
  const float *gates_in = nullptr, *c_prev = nullptr, *h_prev = nullptr;
  float *act = nullptr, *cstate = nullptr, *cact = nullptr, *h = nullptr;
  const uint8_t *zone_state = nullptr, *zone_output = nullptr;
  // backward
  float *dh = nullptr;  // [B, ldh] error on h of step t from above; the error through time is added in place
  const float *b_act = nullptr, *b_cact = nullptr, *b_c_prev = nullptr, *act_next = nullptr, *dgates_next = nullptr, *dc_next = nullptr;
  float *dgates = nullptr, *dcstate = nullptr;
};

// LSTM forward cell for batch row b, cells [c0, c0 + 8), in two halves so that a caller can issue the loads before it
// waits for the recurrent sums: load8 fetches everything the step needs from memory, compute8 takes the recurrent sums
// (rec[8 * g + i] = gate g of cell c0 + i; `first`: the step has no predecessor, cp, hp and rec are zeros).  Same arithmetic,
// in the same order, as lstm_cell_forward_kernel (lstm.cu).
struct LstmForwardIn {
  float gz[8], gi[8], gf[8], go[8], cp[8], hp[8], pi[8], pf[8], po[8];
  unsigned long long zs, zo;
};
// SELF: also fetch what this same cell wrote in the step before (cell state, output); a caller that still holds those
// values in registers passes false and fills in.cp / in.hp itself.  PEEP: fetch the peepholes.
template <bool SELF = true, bool PEEP = true>
__device__ __forceinline__ void lstm_forward_load8(const LstmStep &p, LstmForwardIn &in, long long b, long long c0) {
  const long long C = p.C;
  const float *g = p.gates_in + b * 4 * C + c0;
  load8(in.gz, g); load8(in.gi, g + C); load8(in.gf, g + 2 * C); load8(in.go, g + 3 * C);
  if (SELF) load8(in.cp, p.c_prev + b * C + c0);
  if (PEEP) { load8(in.pi, p.peep + c0); load8(in.pf, p.peep + C + c0); load8(in.po, p.peep + 2 * C + c0); }
  in.zs = p.zone_state != nullptr ? *reinterpret_cast<const unsigned long long *>(p.zone_state + c0) : ~0ull;
  in.zo = p.zone_output != nullptr ? *reinterpret_cast<const unsigned long long *>(p.zone_output + c0) : ~0ull;
  if (SELF && p.zone_output != nullptr) load8(in.hp, p.h_prev + b * p.ldh + c0);
}
struct LstmForwardOut {
  float z[8], ig[8], fg[8], og[8], cs[8], a[8], h[8];
};
__device__ __forceinline__ void lstm_forward_compute8(const LstmForwardIn &in, const float (&rec)[32], bool first, LstmForwardOut &o) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o.z[i] = tanh_ref(in.gz[i] + rec[i]);
    o.ig[i] = sigmoid_ref(in.gi[i] + (rec[8 + i] + in.pi[i] * in.cp[i]));
    o.fg[i] = first ? 0.f : sigmoid_ref(in.gf[i] + rec[16 + i] + in.pf[i] * in.cp[i]);
    float c = o.z[i] * o.ig[i];
    c += o.fg[i] * in.cp[i];
    if (((in.zs >> (8 * i)) & 0xFFull) == 0ull) c = in.cp[i];
    o.cs[i] = c;
    o.a[i] = tanh_ref(c);
    o.og[i] = sigmoid_ref(in.go[i] + rec[24 + i] + in.po[i] * c);
    float hh = o.a[i] * o.og[i];
    if (((in.zo >> (8 * i)) & 0xFFull) == 0ull) hh = in.hp[i];
    o.h[i] = hh;
  }
}
// h is at most 1 in magnitude: its panels have one fixed exponent
constexpr int LSTM_H_EXPONENT = -14;
// what the NEXT step's contraction reads: h as operand panels
__device__ __forceinline__ void lstm_store_h_panels8(const LstmStep &p, const float (&h)[8], long long b, long long c0) {
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = h[i] * 16384.f;
  uint4 h0, h1;
  half_split8(s, h0, h1);
  *reinterpret_cast<uint4 *>(p.p_h0 + b * p.kp + c0) = h0;
  *reinterpret_cast<uint4 *>(p.p_h1 + b * p.kp + c0) = h1;
}
// what the backward pass and the layers above read
__device__ __forceinline__ void lstm_forward_store_arrays8(const LstmStep &p, const LstmForwardOut &o, long long b, long long c0) {
  const long long C = p.C;
  float *act = p.act + b * 4 * C + c0;
  store8(act, o.z); store8(act + C, o.ig); store8(act + 2 * C, o.fg); store8(act + 3 * C, o.og);
  store8(p.cstate + b * C + c0, o.cs);
  store8(p.cact + b * C + c0, o.a);
  store8(p.h + b * p.ldh + c0, o.h);
}
// LSTM backward cell for batch row b, cells [c0, c0 + 8): rec[i] is the error arriving on h of cell c0 + i through time.
// Same arithmetic as lstm_cell_backward_kernel on a step that has a successor; load8 / finish8 as above.
struct LstmBackwardIn {
  float dh[8], z[8], ig[8], fg[8], og[8], a[8], pi[8], pf[8], po[8], cp[8], dni[8], dnf[8], dcn[8], fn[8];
};
// SELF: also fetch what this same cell wrote in the step of the walk before (input / forget gate errors, cell-state
// error); PEEP: fetch the peepholes (see lstm_forward_load8)
template <bool SELF = true, bool PEEP = true>
__device__ __forceinline__ void lstm_backward_load8(const LstmStep &p, LstmBackwardIn &in, long long b, long long c0) {
  const long long C = p.C;
  load8(in.dh, p.dh + b * p.ldh + c0);
  const float *act = p.b_act + b * 4 * C + c0;
  load8(in.z, act); load8(in.ig, act + C); load8(in.fg, act + 2 * C); load8(in.og, act + 3 * C);
  load8(in.a, p.b_cact + b * C + c0);
  if (PEEP) { load8(in.pi, p.peep + c0); load8(in.pf, p.peep + C + c0); load8(in.po, p.peep + 2 * C + c0); }
  if (p.b_c_prev != nullptr) load8(in.cp, p.b_c_prev + b * C + c0);
  if (SELF) {
    const float *dn = p.dgates_next + b * 4 * C + c0;
    load8(in.dni, dn + C); load8(in.dnf, dn + 2 * C);
    load8(in.dcn, p.dc_next + b * C + c0);
  }
  if (p.act_next != nullptr) {
    load8(in.fn, p.act_next + b * 4 * C + 2 * C + c0);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) in.fn[i] = 0.f;
  }
}
struct LstmBackwardOut {
  float dh[8], dz[8], di[8], df[8], d_o[8], dc[8];
};
__device__ __forceinline__ void lstm_backward_compute8(const LstmBackwardIn &in, const float (&rec)[8], bool has_prev, LstmBackwardOut &o) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o.dh[i] = in.dh[i] + rec[i];
    o.d_o[i] = in.og[i] * (1.f - in.og[i]) * (o.dh[i] * in.a[i]);
    float d = o.dh[i] * in.og[i] * (1.f - in.a[i] * in.a[i]);
    d += in.po[i] * o.d_o[i];
    d += in.pi[i] * in.dni[i];
    d += in.pf[i] * in.dnf[i];
    d += in.dcn[i] * in.fn[i];
    o.dc[i] = d;
    o.dz[i] = d * in.ig[i] * (1.f - in.z[i] * in.z[i]);
    o.di[i] = (d * in.z[i]) * (in.ig[i] * (1.f - in.ig[i]));
    o.df[i] = has_prev ? (d * in.cp[i]) * (in.fg[i] * (1.f - in.fg[i])) : 0.f;
  }
}
// the gate errors as operand panels: gate g of the 8 cells at column k0 + 16 g
__device__ __forceinline__ void lstm_store_gate_panels8(const LstmStep &p, const LstmBackwardOut &o, float scale, long long b, long long k0) {
  auto put = [&](const float (&v)[8], int g) {
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = v[i] * scale;
    uint4 h0, h1;
    half_split8(s, h0, h1);
    *reinterpret_cast<uint4 *>(p.p_h0 + b * p.kp + k0 + 16 * g) = h0;
    *reinterpret_cast<uint4 *>(p.p_h1 + b * p.kp + k0 + 16 * g) = h1;
  };
  put(o.dz, 0); put(o.di, 1); put(o.df, 2); put(o.d_o, 3);
}
__device__ __forceinline__ void lstm_backward_store_arrays8(const LstmStep &p, const LstmBackwardOut &o, long long b, long long c0) {
  const long long C = p.C;
  store8(p.dh + b * p.ldh + c0, o.dh);
  float *dg = p.dgates + b * 4 * C + c0;
  store8(dg, o.dz); store8(dg + C, o.di); store8(dg + 2 * C, o.df); store8(dg + 3 * C, o.d_o);
  store8(p.dcstate + b * C + c0, o.dc);
}
}  // namespace myea
