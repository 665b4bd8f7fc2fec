// api.cu -- C ABI of the learned correction's building blocks
// (pmhd_conv3x3, pmhd_conv3x3_wgrad, pmhd_learned_loss_grad; declared in
// include/pmhd.h).
#include <cuda_runtime.h>

#include <condition_variable>
#include <cstdint>
#include <mutex>

#include "learned/conv.h"
#include "learned/net.h"
#include "pmhd.h"

namespace {

// Error words of the convolution calls: host memory the kernels write directly when
// a bounded wait expires, so a call needs no clearing and no copy on the stream --
// one launch and one synchronisation.  One page of ordinary memory, pinned by the
// first call and kept until the process ends: the host may touch it whatever became
// of the device's context, and no thread's start or end allocates or frees pinned
// memory (which would wait for the device and break another thread's capture).
// A call holds one word while it runs.
class ErrorWords {
 public:
  // A cleared word and its device address; nullptr: no pinned memory, or the
  // kernels' shared-memory limits could not be set (once per device and context).
  int* take(int** on_device) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::unique_lock<std::mutex> lock(mu_);
    // A reset context has lost the kernels' limits, so launches fail there until
    // conv_prepare() runs again, and then the page is looked up (and pinned) again too.
    if (prepared_[dev] == 0 || prepared_[dev] != pmhd::learned::conv_prepared()) {
      int** p = &device_page_[dev];
      cudaError_t e = cudaHostGetDevicePointer(p, page_, 0);
      if (e != cudaSuccess) {
        cudaGetLastError();
        e = cudaHostRegister(page_, sizeof(page_), cudaHostRegisterPortable | cudaHostRegisterMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer(p, page_, 0);
      }
      if (e == cudaSuccess) e = pmhd::learned::conv_prepare();
      if (e != cudaSuccess) {
        cudaGetLastError();
        prepared_[dev] = 0;
        return nullptr;
      }
      prepared_[dev] = pmhd::learned::conv_prepared();
    }
    given_back_.wait(lock, [this] { return used_ < kWords; });
    int k = 0;
    while (busy_[k]) k++;
    busy_[k] = true;
    used_++;
    page_[k] = 0;
    *on_device = device_page_[dev] + k;
    return page_ + k;
  }
  void give_back(int* word) {
    bool was_full;
    {
      std::lock_guard<std::mutex> lock(mu_);
      busy_[word - page_] = false;
      was_full = used_-- == kWords;
    }
    if (was_full) given_back_.notify_all();
  }

 private:
  static constexpr int kWords = 1024;
  alignas(4096) int page_[kWords];
  bool busy_[kWords] = {};
  int used_ = 0;
  std::mutex mu_;
  std::condition_variable given_back_;
  int* device_page_[64] = {};
  unsigned prepared_[64] = {};  // conv_prepared() when the device was last looked at, 0: never
};

ErrorWords& error_words() {
  static ErrorWords* words = new ErrorWords;  // outlives the CUDA runtime's own statics
  return *words;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// One synchronous call: launch(error word on the device), wait, status.
template <class Launch>
int call(cudaStream_t s, Launch&& launch) {
  int* on_device = nullptr;
  int* word = error_words().take(&on_device);
  if (!word) return PMHD_ERR_CUDA;
  const cudaError_t e = launch(on_device);
  int rc = PMHD_OK;
  if (e == cudaErrorNotSupported) {
    rc = PMHD_ERR_UNSUPPORTED;
  } else if (e != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    rc = PMHD_ERR_CUDA;
  } else if (*static_cast<const volatile int*>(word)) {
    rc = PMHD_ERR_TIMEOUT;
  }
  error_words().give_back(word);
  return rc;
}

}  // namespace

extern "C" {

int pmhd_conv3x3(int mode, const void* x, int batch, int h, int w, int c_in, const void* weight, const float* bias,
                 int c_out, const void* z_prev, void* out0, void* out1, void* stream) {
  if (batch < 1 || h < 1 || w < 1 || (long long)batch * h * w > (1LL << 31)) return PMHD_ERR_ARG;
  if (!x || !weight || !out0 || !aligned16(x) || !aligned16(weight) || !aligned16(out0)) return PMHD_ERR_ARG;
  if (mode == PMHD_CONV_GELU && (!bias || !out1 || !aligned16(out1))) return PMHD_ERR_ARG;
  if (mode == PMHD_CONV_LINEAR && !bias) return PMHD_ERR_ARG;
  if (mode == PMHD_CONV_DGELU && (!z_prev || !aligned16(z_prev))) return PMHD_ERR_ARG;
  if (mode < PMHD_CONV_GELU || mode > PMHD_CONV_DGELU) return PMHD_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return call(s, [&](int* err) {
    return pmhd::learned::conv3x3(mode, static_cast<const __nv_bfloat16*>(x), batch, h, w, c_in,
                                  static_cast<const __nv_bfloat16*>(weight), bias, c_out,
                                  static_cast<const __nv_bfloat16*>(z_prev), out0, out1, err, s);
  });
}

int pmhd_conv3x3_wgrad(const void* x, const void* dz, int batch, int h, int w, int c_in, int c_out, float* dweight,
                       float* dbias, void* stream) {
  if (batch < 1 || h < 1 || w < 1 || (long long)batch * h * w > (1LL << 31)) return PMHD_ERR_ARG;
  if (!x || !dz || !dweight || !aligned16(x) || !aligned16(dz)) return PMHD_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return call(s, [&](int* err) {
    return pmhd::learned::conv3x3_wgrad(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dz),
                                        batch, h, w, c_in, c_out, dweight, dbias, err, s);
  });
}

int pmhd_learned_loss_grad(const float* out, const float* tgt, int batch, int h, int w, float cx, float cy, void* dz,
                           double* loss, void* stream) {
  if (batch < 1 || h < 1 || w < 1 || (long long)batch * h * w > (1LL << 31)) return PMHD_ERR_ARG;
  if (!out || !tgt || !dz || !loss || !aligned16(dz)) return PMHD_ERR_ARG;
  using namespace pmhd::learned;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Norm hn{};
  hn.cx = cx;
  hn.cy = cy;
  Norm* dn = nullptr;
  float* hist = nullptr;
  int* it = nullptr;
  cudaError_t e = cudaMalloc(&dn, sizeof(Norm));
  if (e == cudaSuccess) e = cudaMalloc(&hist, sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&it, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyAsync(dn, &hn, sizeof(Norm), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(hist, 0, sizeof(float), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(it, 0, sizeof(int), s);
  if (e == cudaSuccess) e = loss_grad(out, tgt, batch, w, h, dn, static_cast<__nv_bfloat16*>(dz), hist, it, s);
  float hl = 0.f;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hl, hist, sizeof(float), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(dn);
  cudaFree(hist);
  cudaFree(it);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return PMHD_ERR_CUDA;
  }
  *loss = hl;
  return PMHD_OK;
}

}  // extern "C"
