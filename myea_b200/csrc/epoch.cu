// The caller of the step: one epoch of mini-batch training and the evaluation pass over a dataset that stays on the
// device.  Replaces Dataset_Mini_Batch::Training_Loop (Dataset__Mini_Batch.cpp:394-436) with Dataset::Train_Batch_BP_Loop
// (Dataset.cpp:667-691) inside it, and the forward-only loop of Dataset::Testing / Measure_Accuracy.
// The reference keeps one row pointer per example ([T * width] floats each) and hands the network a window of those
// pointers; here the rows live in two device arrays and a gather kernel builds each batch in the network's
// [T][B][width] layout from the (host-shuffled) order, so an epoch moves no example over PCIe.
#include "net.cuh"

#include <string.h>

#include <algorithm>

namespace myea {

// One launch gathers the inputs and the targets of a batch straight into the network's buffers:
//   dst[(t * pitch + b) * W + j] = b < B ? src[order[first + b] * T * W + t * W + j] : 0
// (pitch > B: a recurrent network's short batch; its unused rows carry zeros).  V elements per thread and step.
struct GatherSide {
  const float *src;
  float *dst;
  long long W, total;   // total: T * pitch * W / V
};
template <typename V>
__device__ __forceinline__ void gather_side(const GatherSide &g, const unsigned long long *__restrict__ order, long long first, long long B, long long pitch,
                                            long long T, long long i) {
  constexpr int n = sizeof(V) / sizeof(float);
  const long long w = g.W / n, j = i % w, tb = i / w, b = tb % pitch, t = tb / pitch;
  V v = {};
  if (b < B) v = reinterpret_cast<const V *>(g.src)[(order[first + b] * T + t) * w + j];
  reinterpret_cast<V *>(g.dst)[i] = v;
}
__global__ void __launch_bounds__(256) gather_batch_kernel(const GatherSide in, const GatherSide out, int in_vec, int out_vec, const unsigned long long *__restrict__ order,
                                                           long long first, long long B, long long pitch, long long T, int in_blocks) {
  grid_dependency_wait();
  grid_dependency_release();
  const bool is_in = static_cast<int>(blockIdx.x) < in_blocks;
  const GatherSide &g = is_in ? in : out;
  const bool vec = is_in ? in_vec != 0 : out_vec != 0;
  const long long blocks = is_in ? in_blocks : static_cast<long long>(gridDim.x) - in_blocks, block = is_in ? blockIdx.x : static_cast<long long>(blockIdx.x) - in_blocks;
  for (long long i = block * 256ll + threadIdx.x; i < g.total; i += blocks * 256ll) {
    if (vec) gather_side<float4>(g, order, first, B, pitch, T, i);
    else gather_side<float>(g, order, first, B, pitch, T, i);
  }
}

static int gather(myea_b200_net *net, long long first, long long B) {
  Context &ctx = net->ctx;
  const long long pitch = net->full_pitch ? net->B : B;
  auto side = [&](const float *src, float *dst, long long W, int *vec, int *blocks) {
    GatherSide g{src, dst, W, net->T * pitch * W};
    *vec = (W & 3) == 0;
    if (*vec) g.total /= 4;
    *blocks = static_cast<int>(std::max<long long>(1, std::min<long long>((g.total + 255) / 256, 148 * 8)));
    return g;
  };
  int in_vec, out_vec, in_blocks, out_blocks;
  const GatherSide in = side(net->ds_inputs, net->d_input, net->layers[0].n_out, &in_vec, &in_blocks);
  const GatherSide out = side(net->ds_outputs, net->d_desired, net->layers.back().n_out, &out_vec, &out_blocks);
  ctx.begin(TC_ELEMENTWISE);
  launch_dependent(ctx, gather_batch_kernel, dim3(static_cast<unsigned>(in_blocks + out_blocks)), dim3(256), 0, in, out, in_vec, out_vec,
                   static_cast<const unsigned long long *>(net->ds_order), first, B, pitch, net->T, in_blocks);
  ctx.end(TC_ELEMENTWISE);
  return cudaGetLastError() == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}

static int set_order(myea_b200_net *net, const uint64_t *order, uint64_t n) {
  for (uint64_t i = 0; i < n; ++i)
    if (order[i] >= net->ds_examples) { net->ctx.error = "an index of the order is past the end of the dataset"; return MYEA_E_INVALID; }
  if (n > net->ds_order_capacity) {
    if (net->ds_order != nullptr) cudaFree(net->ds_order);
    net->ds_order = nullptr;
    if (cudaMalloc(&net->ds_order, n * sizeof(unsigned long long)) != cudaSuccess) { net->ds_order_capacity = 0; return MYEA_E_CUDA; }
    net->ds_order_capacity = n;
  }
  if (cudaMemcpyAsync(net->ds_order, order, n * sizeof(unsigned long long), cudaMemcpyHostToDevice, net->ctx.stream) != cudaSuccess) return MYEA_E_CUDA;
  return cudaStreamSynchronize(net->ctx.stream) == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;  // `order` is the caller's memory
}

static int reserve_loss_slots(myea_b200_net *net, uint64_t n) {
  if (n > net->ds_loss_capacity) {
    if (net->ds_loss != nullptr) cudaFree(net->ds_loss);
    net->ds_loss = nullptr;
    net->ds_loss_capacity = 0;
    if (cudaMalloc(&net->ds_loss, 3 * n * sizeof(double)) != cudaSuccess) return MYEA_E_CUDA;
    net->ds_loss_capacity = n;
  }
  return cudaMemsetAsync(net->ds_loss, 0, 3 * n * sizeof(double), net->ctx.stream) == cudaSuccess ? MYEA_OK : MYEA_E_CUDA;
}
// points the handle's loss accumulators at the slot of a mini-batch, and back at the end or on the way out
struct LossSlots {
  myea_b200_net *net;
  double *acc;
  unsigned long long *count;
  explicit LossSlots(myea_b200_net *n) : net(n), acc(n->d_loss_acc), count(n->d_loss_count) {}
  void use(uint64_t mb) {
    net->d_loss_acc = net->ds_loss + 3 * mb;
    net->d_loss_count = reinterpret_cast<unsigned long long *>(net->d_loss_acc + 2);
  }
  void restore() { net->d_loss_acc = acc; net->d_loss_count = count; }
  ~LossSlots() { restore(); }
};

// Get__Loss(TYPE_DATASET_NONE) (Neural_Network__Loss.cpp:99-205) of the accumulators of one mini-batch
static double reference_loss(const myea_b200_net *net, double loss_sum, uint64_t number_loss) {
  if (number_loss == 0) return 1.0;
  if (net->desc.type_loss_function == MYEA_LOSS_CROSS_ENTROPY) {
    const uint64_t outputs = static_cast<uint64_t>(net->layers.back().n_out);
    return loss_sum / static_cast<double>(number_loss / outputs);
  }
  return loss_sum / static_cast<double>(number_loss);
}

}  // namespace myea

using namespace myea;

extern "C" int myea_b200_dataset_set(myea_handle net, uint64_t number_examples, const float *inputs, const float *outputs) {
  if (net == nullptr || inputs == nullptr || outputs == nullptr || number_examples == 0) return MYEA_E_INVALID;
  if (cudaSetDevice(net->ctx.device) != cudaSuccess) return MYEA_E_CUDA;
  const size_t wi = static_cast<size_t>(net->T * net->layers[0].n_out), wo = static_cast<size_t>(net->T * net->layers.back().n_out);
  for (float **p : {&net->ds_inputs, &net->ds_outputs}) {
    if (*p != nullptr) cudaFree(*p);
    *p = nullptr;
  }
  net->ds_examples = 0;
  if (cudaMalloc(&net->ds_inputs, number_examples * wi * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&net->ds_outputs, number_examples * wo * sizeof(float)) != cudaSuccess) {
    net->ctx.error = "cudaMalloc failed (dataset)";
    return MYEA_E_CUDA;
  }
  if (cudaMemcpyAsync(net->ds_inputs, inputs, number_examples * wi * sizeof(float), cudaMemcpyHostToDevice, net->ctx.stream) != cudaSuccess ||
      cudaMemcpyAsync(net->ds_outputs, outputs, number_examples * wo * sizeof(float), cudaMemcpyHostToDevice, net->ctx.stream) != cudaSuccess ||
      cudaStreamSynchronize(net->ctx.stream) != cudaSuccess)
    return MYEA_E_CUDA;
  net->ds_examples = number_examples;
  return MYEA_OK;
}

extern "C" int myea_b200_train_epoch(myea_handle net, const uint64_t *order, uint64_t number_examples, uint64_t mini_batch_size,
                                     const myea_opt_desc *opt, uint64_t mask_seed, uint64_t first_step, double *mean_loss, double *accuracy_sum) {
  if (net == nullptr || order == nullptr || opt == nullptr || number_examples == 0) return MYEA_E_INVALID;
  if (net->ds_examples == 0) { net->ctx.error = "no dataset on the device (myea_b200_dataset_set)"; return MYEA_E_INVALID; }
  const uint64_t B = static_cast<uint64_t>(net->B);
  if (mini_batch_size == 0) return MYEA_E_INVALID;
  // Train_Batch_BP walks a mini-batch in sub-batches of the network's batch size, the last one shorter
  // (Dataset.cpp:667-691); the last mini-batch of the epoch may be shorter as well.  Ranks of a data-parallel job take
  // full batches only (see myea_b200_forward).
  if ((mini_batch_size % B != 0 || number_examples % mini_batch_size != 0) && net->comm != nullptr) {
    net->ctx.error = "train_epoch: a multi-GPU network needs a mini-batch that is a multiple of its batch size and divides the number of examples";
    return MYEA_E_UNSUPPORTED;
  }
  // With a communicator the derivative buckets are summed over the ranks inside update_derivative_weight, so a
  // mini-batch is exactly one batch: a second sub-batch would add to sums that have already travelled.
  if (net->comm != nullptr && mini_batch_size != B) {
    net->ctx.error = "train_epoch: with a communicator attached the mini-batch must equal the network's batch size";
    return MYEA_E_UNSUPPORTED;
  }
  if (cudaSetDevice(net->ctx.device) != cudaSuccess) return MYEA_E_CUDA;
  int rc = set_order(net, order, number_examples);
  if (rc != MYEA_OK) return rc;
  const uint64_t mini_batches = (number_examples + mini_batch_size - 1) / mini_batch_size;
  double loss_total = 0.0, acc_total = 0.0;
  // One GPU: every mini-batch accumulates its loss into a slot of its own, and the host reads all of them once at the end -
  // a read per mini-batch would drain the stream each time.  (Ranks of a job add their sums up per mini-batch.)
  const bool slots = net->comm == nullptr;
  if (slots && (rc = reserve_loss_slots(net, mini_batches)) != MYEA_OK) return rc;
  LossSlots slot(net);
  for (uint64_t mb = 0; mb < mini_batches; ++mb) {
    const uint64_t mb_first = mb * mini_batch_size;
    const uint64_t mb_size = std::min<uint64_t>(mini_batch_size, number_examples - mb_first);
    if (mask_seed != 0 && (rc = myea_b200_generate_masks(net, mask_seed, first_step + mb)) != MYEA_OK) return rc;
    if (slots) slot.use(mb);
    else if ((rc = myea_b200_reset_loss(net)) != MYEA_OK) return rc;
    for (uint64_t done = 0; done < mb_size; done += B) {  // derivatives accumulate over the sub-batches of one mini-batch
      const uint64_t b = std::min<uint64_t>(B, mb_size - done);
      const long long first = static_cast<long long>(mb_first + done);
      if ((rc = gather(net, first, static_cast<long long>(b))) != MYEA_OK) return rc;
      if ((rc = net_forward_staged(net, b, 1)) != MYEA_OK) return rc;
      if ((rc = net_error_staged(net, b)) != MYEA_OK) return rc;
      if ((rc = myea_b200_backward(net, b)) != MYEA_OK) return rc;
      if ((rc = myea_b200_update_derivative_weight(net, b)) != MYEA_OK) return rc;
    }
    if (!slots) {
      double ls = 0.0, as = 0.0;
      uint64_t nl = 0;
      if ((rc = myea_b200_get_loss(net, &ls, &nl, &as)) != MYEA_OK) return rc;
      loss_total += reference_loss(net, ls, nl);
      acc_total += as;
    }
    if ((rc = myea_b200_update_parameter(net, mb_size, net->ds_examples, opt)) != MYEA_OK) return rc;
  }
  if (slots) {
    std::vector<double> all(3 * mini_batches);
    slot.restore();
    // the handle's accumulators keep the last mini-batch, as after a loop over the step functions
    if (cudaMemcpyAsync(net->d_loss_acc, net->ds_loss + 3 * (mini_batches - 1), 3 * sizeof(double), cudaMemcpyDeviceToDevice, net->ctx.stream) != cudaSuccess ||
        cudaMemcpyAsync(all.data(), net->ds_loss, all.size() * sizeof(double), cudaMemcpyDeviceToHost, net->ctx.stream) != cudaSuccess ||
        cudaStreamSynchronize(net->ctx.stream) != cudaSuccess)
      return MYEA_E_CUDA;
    for (uint64_t mb = 0; mb < mini_batches; ++mb) {
      uint64_t nl = 0;
      memcpy(&nl, &all[3 * mb + 2], sizeof(nl));
      loss_total += reference_loss(net, all[3 * mb], nl);
      acc_total += all[3 * mb + 1];
    }
  }
  if (mean_loss != nullptr) *mean_loss = loss_total / static_cast<double>(mini_batches);
  if (accuracy_sum != nullptr) *accuracy_sum = acc_total;
  return MYEA_OK;
}

extern "C" int myea_b200_evaluate(myea_handle net, const uint64_t *order, uint64_t number_examples, double *loss, double *loss_sum,
                                  uint64_t *number_loss, double *accuracy_sum) {
  if (net == nullptr || number_examples == 0) return MYEA_E_INVALID;
  if (net->ds_examples == 0) { net->ctx.error = "no dataset on the device (myea_b200_dataset_set)"; return MYEA_E_INVALID; }
  const uint64_t B = static_cast<uint64_t>(net->B);
  if (number_examples % B != 0 && net->comm != nullptr) {
    net->ctx.error = "evaluate: a multi-GPU network needs a number of examples that is a multiple of its batch size";
    return MYEA_E_UNSUPPORTED;
  }
  if (cudaSetDevice(net->ctx.device) != cudaSuccess) return MYEA_E_CUDA;
  std::vector<uint64_t> identity;
  if (order == nullptr) {
    if (number_examples > net->ds_examples) return MYEA_E_INVALID;
    identity.resize(number_examples);
    for (uint64_t i = 0; i < number_examples; ++i) identity[i] = i;
    order = identity.data();
  }
  int rc = set_order(net, order, number_examples);
  if (rc != MYEA_OK) return rc;
  if ((rc = myea_b200_reset_loss(net)) != MYEA_OK) return rc;
  for (uint64_t first = 0; first < number_examples; first += B) {
    const uint64_t b = std::min<uint64_t>(B, number_examples - first);
    if ((rc = gather(net, static_cast<long long>(first), static_cast<long long>(b))) != MYEA_OK) return rc;
    if ((rc = net_forward_staged(net, b, 0)) != MYEA_OK) return rc;   // inference: running statistics, no masks
    if ((rc = net_error_staged(net, b)) != MYEA_OK) return rc;
  }
  double ls = 0.0, as = 0.0;
  uint64_t nl = 0;
  if ((rc = myea_b200_get_loss(net, &ls, &nl, &as)) != MYEA_OK) return rc;
  if (loss != nullptr) *loss = reference_loss(net, ls, nl);
  if (loss_sum != nullptr) *loss_sum = ls;
  if (number_loss != nullptr) *number_loss = nl;
  if (accuracy_sum != nullptr) *accuracy_sum = as;
  return MYEA_OK;
}
