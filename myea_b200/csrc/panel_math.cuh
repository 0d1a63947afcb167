// The arithmetic of one LSTM cell step for 8 consecutive cells of one batch row, and how its results leave as operand panels
// of the next step (lstm_persistent.cu); the activation functions as lstm.cu has them.
#pragma once

#include "common.cuh"
#include "half_panels.cuh"

namespace myea {

// 32 aligned bytes in one access
__device__ __forceinline__ void load32(float (&d)[8], const float *p) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void store32(float *p, const float (&d)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(d[0]), "f"(d[1]), "f"(d[2]), "f"(d[3]), "f"(d[4]), "f"(d[5]), "f"(d[6]),
               "f"(d[7])
               : "memory");
}
// 1 / d for d in [1, inf], without a branch, so that the eight cells of a thread interleave: the hardware's approximation and one
// Newton-Raphson step in fused arithmetic (P. Markstein, IA-64 and Elementary Functions, 2000).  The theorem there does not cover
// every d: tests/test_small_shapes_gpu.py compares all of [1, 2^126) with __frcp_rn, and none of the 1056964608 differs.
// Past 2^126 the approximation stands (0 where the reciprocal is at most 1.2e-38).
__device__ __forceinline__ float reciprocal_from_one(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float n = fmaf(r, fmaf(-d, r, 1.0f), r);
  return d < 8.507059e37f ? n : r;
}
// the gates' functions as the reference has them (Activation_Functions.hpp:40, :45): 1 / (1 + e^-x), 2 / (1 + e^-2x) - 1
__device__ __forceinline__ float sigmoid_cell(float x) { return reciprocal_from_one(1.0f + expf(-x)); }
__device__ __forceinline__ float tanh_cell(float x) { return 2.0f * reciprocal_from_one(1.0f + expf(-2.0f * x)) - 1.0f; }

// One time step of an LSTM layer as the cell arithmetic sees it: the arrays of step t, of the step before / after it in
// the layer's direction, and where the results also leave as operand panels of the next step's contraction.
struct LstmStep {
  long long C = 0, ldh = 0, kp = 0;
  uint16_t *p_h0 = nullptr, *p_h1 = nullptr;  // operand panels written for the next step (pitch kp), or null
  // forward (rows of step t unless said otherwise)
  const float *gates_in = nullptr;
  float *act = nullptr, *cstate = nullptr, *cact = nullptr, *h = nullptr;
  const uint8_t *zone_state = nullptr, *zone_output = nullptr;
  // backward
  float *dh = nullptr;  // [B, ldh] error on h of step t from above; the error through time is added in place
  const float *b_act = nullptr, *b_cact = nullptr, *b_c_prev = nullptr;
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
// (what this same cell computed in the step before, in.cp and in.hp, and the peepholes stay with the caller)
__device__ __forceinline__ void lstm_forward_load8(const LstmStep &p, LstmForwardIn &in, long long b, long long c0) {
  const long long C = p.C;
  const float *g = p.gates_in + b * 4 * C + c0;
  load32(in.gz, g); load32(in.gi, g + C); load32(in.gf, g + 2 * C); load32(in.go, g + 3 * C);
  in.zs = p.zone_state != nullptr ? *reinterpret_cast<const unsigned long long *>(p.zone_state + c0) : ~0ull;
  in.zo = p.zone_output != nullptr ? *reinterpret_cast<const unsigned long long *>(p.zone_output + c0) : ~0ull;
}
struct LstmForwardOut {
  float z[8], ig[8], fg[8], og[8], cs[8], a[8], h[8];
};
__device__ __forceinline__ void lstm_forward_compute8(const LstmForwardIn &in, const float (&rec)[32], bool first, LstmForwardOut &o) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o.z[i] = tanh_cell(in.gz[i] + rec[i]);
    o.ig[i] = sigmoid_cell(in.gi[i] + (rec[8 + i] + in.pi[i] * in.cp[i]));
    o.fg[i] = first ? 0.f : sigmoid_cell(in.gf[i] + rec[16 + i] + in.pf[i] * in.cp[i]);
    float c = o.z[i] * o.ig[i];
    c += o.fg[i] * in.cp[i];
    if (((in.zs >> (8 * i)) & 0xFFull) == 0ull) c = in.cp[i];
    o.cs[i] = c;
    o.a[i] = tanh_cell(c);
    o.og[i] = sigmoid_cell(in.go[i] + rec[24 + i] + in.po[i] * c);
    float hh = o.a[i] * o.og[i];
    if (((in.zo >> (8 * i)) & 0xFFull) == 0ull) hh = in.hp[i];
    o.h[i] = hh;
  }
}
// h is at most 1 in magnitude and known to 2^-24 of that (tanh_cell is a difference from 1): its panels have one fixed exponent and a
// step of 2^-39
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
constexpr int LSTM_FORWARD_ARRAYS = 7, LSTM_BACKWARD_ARRAYS = 6;
__device__ __forceinline__ void lstm_forward_store_array8(const LstmStep &p, const LstmForwardOut &o, long long b, long long c0, int k) {
  const long long C = p.C;
  float *act = p.act + b * 4 * C + c0;
  switch (k) {
    case 0: store32(act, o.z); break;
    case 1: store32(act + C, o.ig); break;
    case 2: store32(act + 2 * C, o.fg); break;
    case 3: store32(act + 3 * C, o.og); break;
    case 4: store32(p.cstate + b * C + c0, o.cs); break;
    case 5: store32(p.cact + b * C + c0, o.a); break;
    default: store32(p.h + b * p.ldh + c0, o.h); break;
  }
}
// LSTM backward cell for batch row b, cells [c0, c0 + 8): rec[i] is the error arriving on h of cell c0 + i through time.
// Same arithmetic as lstm_cell_backward_kernel on a step that has a successor; load8 / finish8 as above.
struct LstmBackwardIn {
  float dh[8], z[8], ig[8], fg[8], og[8], a[8], pi[8], pf[8], po[8], cp[8], dni[8], dnf[8], dcn[8], fn[8];
};
// (dni, dnf, dcn and fn, the step of the walk before, and the peepholes stay with the caller)
__device__ __forceinline__ void lstm_backward_load8(const LstmStep &p, LstmBackwardIn &in, long long b, long long c0) {
  const long long C = p.C;
  load32(in.dh, p.dh + b * p.ldh + c0);
  const float *act = p.b_act + b * 4 * C + c0;
  load32(in.z, act); load32(in.ig, act + C); load32(in.fg, act + 2 * C); load32(in.og, act + 3 * C);
  load32(in.a, p.b_cact + b * C + c0);
  if (p.b_c_prev != nullptr) load32(in.cp, p.b_c_prev + b * C + c0);
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
__device__ __forceinline__ void lstm_backward_store_array8(const LstmStep &p, const LstmBackwardOut &o, long long b, long long c0, int k) {
  const long long C = p.C;
  float *dg = p.dgates + b * 4 * C + c0;
  switch (k) {
    case 0: store32(p.dh + b * p.ldh + c0, o.dh); break;
    case 1: store32(dg, o.dz); break;
    case 2: store32(dg + C, o.di); break;
    case 3: store32(dg + 2 * C, o.df); break;
    case 4: store32(dg + 3 * C, o.d_o); break;
    default: store32(p.dcstate + b * C + c0, o.dc); break;
  }
}
}  // namespace myea
