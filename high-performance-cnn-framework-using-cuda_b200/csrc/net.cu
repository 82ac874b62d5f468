// Fused-network handle: parameter arena, status word and options.
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "net.cuh"

namespace cnn {
void destroy_host_pipeline(HostPipeline* p);

// One allocation, in the first training call of a net.  (One row per SM: no gradient kernel has more blocks.)
int ensure_train_scratch(cnn_net* net) {
  if (net->d_grad) return CNN_OK;
  constexpr size_t kGrad = kNParamsPadded + 32;
  CNN_CUDA(cudaMalloc(&net->d_grad, sizeof(float) * (kGrad + (size_t)kRowStride * sm_count())));
  net->d_partials = net->d_grad + kGrad;
  return CNN_OK;
}
}  // namespace cnn

using namespace cnn;

extern "C" {

int cnn_net_create(unsigned int seed, cnn_net** out) {
  CNN_REQUIRE(out != nullptr, "cnn_net_create: out is NULL");
  *out = nullptr;
  cnn_net* net = new (std::nothrow) cnn_net();
  CNN_REQUIRE(net != nullptr, "cnn_net_create: out of host memory");
  net->seed = seed;
  cudaError_t e = cudaGetDevice(&net->device);
  if (e == cudaSuccess) e = cudaMalloc(&net->d_params, sizeof(float) * kNParamsPadded);
  const size_t status_bytes = sizeof(GradLeft) * (1 + (size_t)sm_count());      // status word, length of the queue, and the queue of GradLeft
  if (e == cudaSuccess) e = cudaMalloc(&net->d_status, status_bytes);
  if (e == cudaSuccess) e = cudaMemset(net->d_status, 0, status_bytes);
  if (e != cudaSuccess) {
    cnn_net_destroy(net);
    return cuda_fail(e, "cnn_net_create");
  }
  // Draw order of the reference's static Layer objects (main.cu:18-20 through layer.cu:19-27):
  // c1 (6 units: bias, 25 weights), s1 (1 unit: bias, 16 weights), f (10 units: bias, 216 weights).
  std::vector<float> h(kNParamsPadded, 0.f);
  srand(seed);
  auto draw = [] { return 0.5f - float(rand()) / float(RAND_MAX); };
  for (int i = 0; i < kF; ++i) {
    h[kOffBc + i] = draw();
    for (int j = 0; j < 25; ++j) h[kOffWc + i * 25 + j] = draw();
  }
  h[kOffBs] = draw();
  for (int j = 0; j < 16; ++j) h[kOffWs + j] = draw();
  for (int i = 0; i < kOut; ++i) {
    h[kOffBf + i] = draw();
    for (int j = 0; j < kS; ++j) h[kOffWf + i * kS + j] = draw();
  }
  e = cudaMemcpy(net->d_params, h.data(), sizeof(float) * kNParamsPadded, cudaMemcpyHostToDevice);
  // the upload and the status memset must have landed before a launch on a non-blocking stream
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cnn_net_destroy(net);
    return cuda_fail(e, "cnn_net_create: parameter upload");
  }
  *out = net;
  return CNN_OK;
}

int cnn_net_destroy(cnn_net* net) {
  if (!net) return CNN_OK;
  cudaFree(net->d_params);
  cudaFree(net->d_status);
  cudaFree(net->d_grad);      // and d_partials behind it
  destroy_host_pipeline(net->host);
  delete net;
  return CNN_OK;
}

int cnn_net_set_params(cnn_net* net, const float* h_params) {
  CNN_REQUIRE(net && h_params, "cnn_net_set_params: NULL argument");
  // Wait for work in flight that may still read the old values, upload, and wait again: a copy from
  // pageable memory may return while its DMA is pending, and a launch on a non-blocking stream (the
  // host pipeline's, or the caller's) is not ordered behind it.
  CNN_CUDA(cudaDeviceSynchronize());
  CNN_CUDA(cudaMemcpy(net->d_params, h_params, sizeof(float) * kNParams, cudaMemcpyHostToDevice));
  CNN_CUDA(cudaDeviceSynchronize());
  return CNN_OK;
}

int cnn_net_get_params(cnn_net* net, float* h_params) {
  CNN_REQUIRE(net && h_params, "cnn_net_get_params: NULL argument");
  CNN_CUDA(cudaMemcpy(h_params, net->d_params, sizeof(float) * kNParams, cudaMemcpyDeviceToHost));
  return CNN_OK;
}

int cnn_net_params_device(cnn_net* net, float** d_params) {
  CNN_REQUIRE(net && d_params, "cnn_net_params_device: NULL argument");
  *d_params = net->d_params;
  return CNN_OK;
}

int cnn_net_set_fast_sigmoid(cnn_net* net, int enable) {
  CNN_REQUIRE(net, "cnn_net_set_fast_sigmoid: NULL net");
  net->fast_sigmoid = enable ? 1 : 0;
  return CNN_OK;
}

int cnn_net_set_option(cnn_net* net, const char* key, int value) {
  CNN_REQUIRE(net && key, "cnn_net_set_option: NULL argument");
  if (std::strcmp(key, "persample_kernel") == 0) {
    CNN_REQUIRE(value == 0 || value == 1, "cnn_net_set_option: persample_kernel takes 0 or 1");
    net->ps_kernel = value;
    return CNN_OK;
  }
  if (std::strcmp(key, "forward_path") == 0) {
    CNN_REQUIRE(value >= -1 && value <= 2, "cnn_net_set_option: forward_path takes -1 (by batch size), 0, 1 or 2");
    net->forward_path = value;
    return CNN_OK;
  }
  if (std::strcmp(key, "grad_path") == 0) {
    CNN_REQUIRE(value >= -1 && value <= 1, "cnn_net_set_option: grad_path takes -1 (by batch size), 0 or 1");
    net->grad_path = value;
    return CNN_OK;
  }
  if (std::strcmp(key, "fast_sigmoid") == 0) {
    net->fast_sigmoid = value ? 1 : 0;
    return CNN_OK;
  }
  set_error("cnn_net_set_option: unknown option '%s'", key);
  return CNN_ERR_INVALID;
}

int cnn_net_status(cnn_net* net, int* status) {
  CNN_REQUIRE(net && status, "cnn_net_status: NULL argument");
  CNN_CUDA(cudaDeviceSynchronize());
  CNN_CUDA(cudaMemcpy(status, net->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  if (*status != 0) {
    set_error("a bounded device-side wait ran out (status %d)", *status);
    int zero = 0;
    CNN_CUDA(cudaMemcpy(net->d_status, &zero, sizeof(int), cudaMemcpyHostToDevice));
    return CNN_ERR_TIMEOUT;
  }
  return CNN_OK;
}

}  // extern "C"
