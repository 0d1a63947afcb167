// One fused parameter update over the flat parameter buffer, the global-norm clip that precedes it and the
// derivative reset that follows it: Update_Parameters__Adam (Neural_Network__Adam.cpp:39-95), AMSGrad
// (Neural_Network__AMSGrad.cpp), AdaBound / AMSBound (Neural_Network__AdaBound.cpp, …AMSBound.cpp), gradient descent,
// momentum and Nesterov (Neural_Network__Gradient_Descent.cpp, …_Momentum.cpp, Neural_Network__Nesterov_Accelerated_Gradient.cpp), iRPROP+
// (Neural_Network__iRPROP_plus.cpp),
// Clip_Gradient / Euclidean_Norm (Neural_Network__Clip_Gradient.cpp:82-94, …Regularization__Max_Norm_Constraints.cpp:48-87).
// Pure HBM streaming: every array is read and written once with 128-bit accesses; the optimizer is a uniform branch.
#include "common.cuh"
#include "half_panels.cuh"

#include <algorithm>

namespace myea {

__device__ __forceinline__ float opt_one(const OptLaunch &o, float w, float g, float &m, float &v, float &vhat, float &prev, float mask) {
  const float decay = (o.weight_decay != 0.f) ? mask * o.weight_decay * w : 0.f;
  switch (o.type) {
    case MYEA_OPT_ADAM: {
      m = o.beta1 * m + (1.f - o.beta1) * g;
      v = o.beta2 * v + (1.f - o.beta2) * g * g;
      return w - (o.lr_t * m / (sqrtf(v) + o.epsilon) + decay);
    }
    case MYEA_OPT_AMSGRAD: {
      m = o.beta1 * m + (1.f - o.beta1) * g;
      v = o.beta2 * v + (1.f - o.beta2) * g * g;
      vhat = fmaxf(vhat, v);
      return w - (o.lr_t * m / (sqrtf(vhat) + o.epsilon) + decay);
    }
    case MYEA_OPT_ADABOUND: {
      m = o.beta1 * m + (1.f - o.beta1) * g;
      v = o.beta2 * v + (1.f - o.beta2) * g * g;
      const float step = fminf(fmaxf(o.lr_t / (sqrtf(v) + o.epsilon), o.lower), o.upper);
      return w - (step * m + decay);
    }
    case MYEA_OPT_AMSBOUND: {
      m = o.beta1 * m + (1.f - o.beta1) * g;
      v = o.beta2 * v + (1.f - o.beta2) * g * g;
      vhat = fmaxf(vhat, v);
      const float step = fminf(fmaxf(o.lr_t / (sqrtf(vhat) + o.epsilon), o.lower), o.upper);
      return w - (step * m + decay);
    }
    case MYEA_OPT_IRPROP_PLUS: {
      // Update_Parameter__iRPROP_plus__Loop (Neural_Network__iRPROP_plus.cpp:30-120).  m: previous derivative,
      // v: previous step (a cleared 0 stands for rprop_delta_zero, Clear_Optimizer, Train.cpp:163-190), prev: previous
      // delta weight.  No decay term: the reference has none on this path.
      if (v == 0.f) v = o.rprop_zero;
      const float same = m * g;
      const float sign = static_cast<float>(0.f < g) - static_cast<float>(g < 0.f);
      if (same > 0.f) {
        v = fminf(v * o.rprop_increase, o.rprop_max);
        prev = -sign * v;
        m = g;
        return w + prev;
      }
      if (same < 0.f) {
        v = fmaxf(v * o.rprop_decrease, o.rprop_min);
        m = 0.f;
        return o.rprop_error_is_worse ? w - prev : w;
      }
      prev = -sign * v;
      m = g;
      return w + prev;
    }
    default: {  // gradient descent family
      if (o.momentum == 0.f) return w - (o.gd_lr * g + decay);
      if (!o.nesterov) {
        // delta = lr*g + momentum*previous delta ; w -= delta
        const float delta = o.gd_lr * g + o.momentum * prev;
        prev = delta;
        return w - (delta + decay);
      }
      // Nesterov exactly as the reference codes it (Neural_Network__Nesterov_Accelerated_Gradient.cpp:48,59):
      // delta = lr*g + momentum*previous delta ; w -= momentum*delta - lr*g
      const float delta = o.gd_lr * g + o.momentum * prev;
      prev = delta;
      return w - (o.momentum * delta - o.gd_lr * g + decay);
    }
  }
}

template <bool HAS_VHAT, bool HAS_PREV>
__global__ void __launch_bounds__(256) optimizer_kernel(const OptLaunch o, const OptArrays a, size_t n) {
  grid_dependency_wait();
  grid_dependency_release();
  const float scale = o.clip_scale != nullptr ? *o.clip_scale : 1.0f;
  const size_t n4 = n >> 2;
  const bool adam_like = o.type != MYEA_OPT_GD;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float4 w = reinterpret_cast<float4 *>(a.w)[i];
    float4 g = reinterpret_cast<float4 *>(a.g)[i];
    float4 m = make_float4(0, 0, 0, 0), v = m, vh = m, pv = m, mk = make_float4(1, 1, 1, 1);
    if (adam_like) { m = reinterpret_cast<float4 *>(a.m)[i]; v = reinterpret_cast<float4 *>(a.v)[i]; }
    if (HAS_VHAT) vh = reinterpret_cast<float4 *>(a.vhat)[i];
    if (HAS_PREV) pv = reinterpret_cast<float4 *>(a.prev)[i];
    if (o.weight_decay != 0.f && a.mask != nullptr) mk = reinterpret_cast<const float4 *>(a.mask)[i];
    w.x = opt_one(o, w.x, g.x * scale, m.x, v.x, vh.x, pv.x, mk.x);
    w.y = opt_one(o, w.y, g.y * scale, m.y, v.y, vh.y, pv.y, mk.y);
    w.z = opt_one(o, w.z, g.z * scale, m.z, v.z, vh.z, pv.z, mk.z);
    w.w = opt_one(o, w.w, g.w * scale, m.w, v.w, vh.w, pv.w, mk.w);
    reinterpret_cast<float4 *>(a.w)[i] = w;
    reinterpret_cast<float4 *>(a.g)[i] = make_float4(0, 0, 0, 0);
    if (adam_like) { reinterpret_cast<float4 *>(a.m)[i] = m; reinterpret_cast<float4 *>(a.v)[i] = v; }
    if (HAS_VHAT) reinterpret_cast<float4 *>(a.vhat)[i] = vh;
    if (HAS_PREV) reinterpret_cast<float4 *>(a.prev)[i] = pv;
  }
  // tail (n not a multiple of 4)
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const size_t i = (n4 << 2) + threadIdx.x;
    float m = adam_like ? a.m[i] : 0.f, v = adam_like ? a.v[i] : 0.f, vh = HAS_VHAT ? a.vhat[i] : 0.f, pv = HAS_PREV ? a.prev[i] : 0.f;
    const float mk = (o.weight_decay != 0.f && a.mask != nullptr) ? a.mask[i] : 1.f;
    a.w[i] = opt_one(o, a.w[i], a.g[i] * scale, m, v, vh, pv, mk);
    a.g[i] = 0.f;
    if (adam_like) { a.m[i] = m; a.v[i] = v; }
    if (HAS_VHAT) a.vhat[i] = vh;
    if (HAS_PREV) a.prev[i] = pv;
  }
}

static bool opt_arrays(const OptLaunch &o, const OptArrays &a, bool &has_vhat, bool &has_prev) {
  has_vhat = (o.type == MYEA_OPT_AMSGRAD || o.type == MYEA_OPT_AMSBOUND);
  has_prev = (o.type == MYEA_OPT_GD && o.momentum != 0.f) || o.type == MYEA_OPT_IRPROP_PLUS;
  return !((has_vhat && a.vhat == nullptr) || (has_prev && a.prev == nullptr) || (o.type != MYEA_OPT_GD && (a.m == nullptr || a.v == nullptr)));
}

int optimizer_update(Context &ctx, const OptLaunch &o, const OptArrays &a, size_t n) {
  bool has_vhat, has_prev;
  if (!opt_arrays(o, a, has_vhat, has_prev)) return MYEA_E_INVALID;
  const int blocks = static_cast<int>(std::max<size_t>(1, std::min<size_t>(((n >> 2) + 255) / 256, 148 * 16)));
  ctx.begin(TC_OPTIMIZER);
  if (has_vhat) launch_dependent(ctx, optimizer_kernel<true, false>, dim3(blocks), dim3(256), 0, o, a, n);
  else if (has_prev) launch_dependent(ctx, optimizer_kernel<false, true>, dim3(blocks), dim3(256), 0, o, a, n);
  else launch_dependent(ctx, optimizer_kernel<false, false>, dim3(blocks), dim3(256), 0, o, a, n);
  ctx.end(TC_OPTIMIZER);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// The update of weights that contractions read as operand panels: a CTA updates a block of 128 x 128 weights, keeps the new
// values, finds the exponents of their rows and columns and writes the panels of the next step along, which otherwise cost a pass
// of their own over the weights (4 bytes read and 8 written per weight); the derivatives are not zeroed (4 bytes less), the next accumulation
// overwrites them instead of adding to them (4 bytes less again).  Bound by HBM, so by loads in flight: a thread has 8 elements
// of all arrays on the way, 1024 threads per SM; the new weights wait in shared memory (64 KB) because in registers they leave
// room for half the threads (138 M weights, Adam: 764 us, 36 bytes per weight at 6.5 TB/s; with the weights in registers and 512
// threads per SM 1770 us at 32 bytes per weight).  Behind contractions that hold the chip at its power cap it takes
// 950 us, with or without its arithmetic, and in proportion without its panels: memory at the clocks that are left.
constexpr int OPT_LAYERS = 32;
constexpr int OPT_THREADS = HP_THREADS, OPT_ROWS = HP_ROWS;   // 8 columns of rows tid / 16 + 32 i
constexpr int OPT_SMEM = HP_BLOCK * HP_BLOCK * 4;
struct OptPanelTable {
  OptPanelLayer l[OPT_LAYERS];
  int n;
};
template <bool HAS_VHAT, bool HAS_PREV>
__global__ void __launch_bounds__(OPT_THREADS, 2) optimizer_panels_kernel(const OptLaunch o, const OptArrays a, const __grid_constant__ OptPanelTable t) {
  extern __shared__ float4 kept[];   // [row][2][thread]
  grid_dependency_wait();
  grid_dependency_release();
  const float scale = o.clip_scale != nullptr ? *o.clip_scale : 1.0f;
  const bool adam_like = o.type != MYEA_OPT_GD, decays = o.weight_decay != 0.f && a.mask != nullptr;
  int k = 0;
  while (k + 1 < t.n && static_cast<int>(blockIdx.x) >= t.l[k + 1].first_block) ++k;
  const HalfPanels &p = t.l[k].p;
  const int block = static_cast<int>(blockIdx.x) - t.l[k].first_block;
  const int across = static_cast<int>((p.C + HP_BLOCK - 1) / HP_BLOCK), by = block / across, bx = block - by * across;
  const long long c = bx * static_cast<long long>(HP_BLOCK) + (threadIdx.x & 15) * 8;
  const long long r0 = by * static_cast<long long>(HP_BLOCK) + (threadIdx.x >> 4);
#pragma unroll 1
  for (int i = 0; i < OPT_ROWS; ++i) {
    const long long r = r0 + OPT_THREADS / 16 * i;
    float w[8] = {};
    if (r < p.R && c < p.C) {
      const size_t at = t.l[k].offset + static_cast<size_t>(r * p.C + c);
      float g[8], m[8] = {}, v[8] = {}, vh[8] = {}, pv[8] = {}, mk[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
      ld8(w, a.w + at, 8, true);
      ld8(g, a.g + at, 8, true);
      if (adam_like) { ld8(m, a.m + at, 8, true); ld8(v, a.v + at, 8, true); }
      if (HAS_VHAT) ld8(vh, a.vhat + at, 8, true);
      if (HAS_PREV) ld8(pv, a.prev + at, 8, true);
      if (decays) ld8(mk, a.mask + at, 8, true);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = opt_one(o, w[j], g[j] * scale, m[j], v[j], vh[j], pv[j], mk[j]);
      st8(a.w + at, w, 8, true);
      if (adam_like) { st8(a.m + at, m, 8, true); st8(a.v + at, v, 8, true); }
      if (HAS_VHAT) st8(a.vhat + at, vh, 8, true);
      if (HAS_PREV) st8(a.prev + at, pv, 8, true);
    }
    kept[(2 * i) * OPT_THREADS + threadIdx.x] = make_float4(w[0], w[1], w[2], w[3]);
    kept[(2 * i + 1) * OPT_THREADS + threadIdx.x] = make_float4(w[4], w[5], w[6], w[7]);
  }
  float v[OPT_ROWS][8];
#pragma unroll
  for (int i = 0; i < OPT_ROWS; ++i) {
    const float4 x = kept[(2 * i) * OPT_THREADS + threadIdx.x], y = kept[(2 * i + 1) * OPT_THREADS + threadIdx.x];
    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w; v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
  }
  half_store_block(p, by, bx, v);
}
template <bool HAS_VHAT, bool HAS_PREV>
static int launch_optimizer_panels(Context &ctx, int blocks, const OptLaunch &o, const OptArrays &a, const OptPanelTable &t) {
  auto kernel = optimizer_panels_kernel<HAS_VHAT, HAS_PREV>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OPT_SMEM) != cudaSuccess) return MYEA_E_CUDA;
  return launch_dependent(ctx, kernel, dim3(blocks), dim3(OPT_THREADS), OPT_SMEM, o, a, t) == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

int optimizer_update_panels(Context &ctx, const OptLaunch &o, const OptArrays &a, const OptPanelLayer *layers, int n) {
  bool has_vhat, has_prev;
  if (!opt_arrays(o, a, has_vhat, has_prev)) return MYEA_E_INVALID;
  for (int first = 0; first < n; first += OPT_LAYERS) {
    OptPanelTable t = {};
    t.n = std::min(OPT_LAYERS, n - first);
    int blocks = 0;
    for (int k = 0; k < t.n; ++k) {
      t.l[k] = layers[first + k];
      t.l[k].first_block = blocks;
      blocks += static_cast<int>(((t.l[k].p.R + HP_BLOCK - 1) / HP_BLOCK) * ((t.l[k].p.C + HP_BLOCK - 1) / HP_BLOCK));
    }
    ctx.begin(TC_OPTIMIZER);
    const int rc = has_vhat ? launch_optimizer_panels<true, false>(ctx, blocks, o, a, t)
                 : has_prev ? launch_optimizer_panels<false, true>(ctx, blocks, o, a, t) : launch_optimizer_panels<false, false>(ctx, blocks, o, a, t);
    ctx.end(TC_OPTIMIZER);
    if (rc != MYEA_OK) return rc;
  }
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// sum of squares of the whole derivative buffer, double accumulation across blocks
__global__ void __launch_bounds__(256) sum_squares_kernel(const float *__restrict__ g, size_t n, double *out) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ float sh[8];
  float s = 0.f;
  const size_t n4 = n >> 2;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const float4 t = reinterpret_cast<const float4 *>(g)[i];
    s += t.x * t.x + t.y * t.y + t.z * t.z + t.w * t.w;
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) { const float t = g[(n4 << 2) + threadIdx.x]; s += t * t; }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += static_cast<double>(sh[w]);
    atomicAdd(out, t);
  }
}

int sum_squares(Context &ctx, const float *g, size_t n, double *d_out, bool accumulate) {
  ctx.begin(TC_OPTIMIZER);
  if (!accumulate) cudaMemsetAsync(d_out, 0, sizeof(double), ctx.stream);
  const int blocks = static_cast<int>(std::max<size_t>(1, std::min<size_t>(((n >> 2) + 255) / 256, 148 * 8)));
  launch_dependent(ctx, sum_squares_kernel, dim3(blocks), dim3(256), 0, g, n, d_out);
  ctx.end(TC_OPTIMIZER);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

__global__ void clip_scale_kernel(const double *sumsq, float clip, float *scale) {
  grid_dependency_wait();
  grid_dependency_release();
  const float norm = sqrtf(static_cast<float>(*sumsq));
  *scale = norm >= clip ? clip / norm : 1.0f;
}

int clip_scale_from_norm(Context &ctx, const double *d_sumsq, float clip, float *d_scale) {
  launch_dependent(ctx, clip_scale_kernel, dim3(1), dim3(1), 0, d_sumsq, clip, d_scale);
  ctx.launches += 1;
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

// one block per row: sum of squares (fp32 partials, tree), then the scale
__global__ void __launch_bounds__(256) row_max_norm_kernel(float *__restrict__ w, long long cols, float max_norm) {
  __shared__ float sh[256];
  float *row = w + static_cast<long long>(blockIdx.x) * cols;
  float acc = 0.f;
  for (long long j = threadIdx.x; j < cols; j += blockDim.x) acc = fmaf(row[j], row[j], acc);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  const float norm = sqrtf(sh[0]);
  if (norm >= max_norm) {
    const float scale = max_norm / norm;
    for (long long j = threadIdx.x; j < cols; j += blockDim.x) row[j] *= scale;
  }
}

// LSTM blocks (Update_Weight_Regularization__Max_Norm_Constraints__LSTMs, …Max_Norm_Constraints.cpp:167-310): every run
// of weights is a vector of its own - per cell the input and the recurrent weights of the cell input, per block those
// of the three gates, and the three peephole runs.  One thread block per run: grid (blocks of the layer, 2 cpb + 9).
// The reference tests `first_index > start` with start = 0: a run that begins at parameter 0 is passed over.
__global__ void __launch_bounds__(256) lstm_max_norm_kernel(float *__restrict__ params, long long first, long long stride, long long I, long long C,
                                                            long long cpb, float max_norm) {
  __shared__ float sh[256];
  const long long s = blockIdx.y, base = first + static_cast<long long>(blockIdx.x) * stride;
  long long at, len;
  if (s < 2 * cpb) {
    at = base + (s >> 1) * (I + C) + ((s & 1) ? I : 0);
    len = (s & 1) ? C : I;
  } else {
    const long long g = s - 2 * cpb, g0 = base + cpb * (I + C);
    if (g < 3) { at = g0 + g * I; len = I; }
    else if (g < 6) { at = g0 + 3 * I + (g - 3) * C; len = C; }
    else { at = g0 + 3 * I + 3 * C + (g - 6) * cpb; len = cpb; }
  }
  if (at == 0) return;
  float *v = params + at;
  float acc = 0.f;
  for (long long j = threadIdx.x; j < len; j += blockDim.x) acc = fmaf(v[j], v[j], acc);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  const float norm = sqrtf(sh[0]);
  if (norm >= max_norm) {
    const float scale = max_norm / norm;
    for (long long j = threadIdx.x; j < len; j += blockDim.x) v[j] *= scale;
  }
}

int lstm_max_norm(Context &ctx, float *params, long long first, long long blocks, long long stride, long long n_in, long long cells,
                  long long cells_per_block, float max_norm) {
  if (blocks <= 0) return MYEA_OK;
  ctx.begin(TC_OPTIMIZER);
  lstm_max_norm_kernel<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(2 * cells_per_block + 9)), 256, 0, ctx.stream>>>(
      params, first, stride, n_in, cells, cells_per_block, max_norm);
  ctx.end(TC_OPTIMIZER);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

int row_max_norm(Context &ctx, float *w, long long rows, long long cols, float max_norm) {
  if (rows <= 0 || cols <= 0) return MYEA_OK;
  ctx.begin(TC_OPTIMIZER);
  row_max_norm_kernel<<<static_cast<unsigned>(rows), 256, 0, ctx.stream>>>(w, cols, max_norm);
  ctx.end(TC_OPTIMIZER);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

}  // namespace myea
