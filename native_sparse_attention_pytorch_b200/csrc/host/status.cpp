// A copy of a device status word on its way to the host: started after some call, looked at during a later one.

#include <cuda_runtime_api.h>

#include <atomic>

#include "nsa_host.h"

namespace nsa_host {

static std::atomic<bool> g_backward_ran[C10_COMPILE_TIME_MAX_GPUS];

void note_backward(const Tensor& t) { g_backward_ran[t.get_device()].store(true, std::memory_order_release); }

class StatusCopy {
 public:
  // `word` [1]: the device's status word; the event belongs to its device, whichever is current
  explicit StatusCopy(const Tensor& word) : device_(word.device()) {
    require_cuda(word);
    const c10::cuda::CUDAGuard guard(device_);
    if (cudaHostAlloc(reinterpret_cast<void**>(&word_), sizeof(int32_t), cudaHostAllocPortable) != cudaSuccess ||
        cudaEventCreateWithFlags(&event_, cudaEventDisableTiming) != cudaSuccess)
      throw Error("status poll: no pinned word or event");
    *word_ = 0;
  }
  ~StatusCopy() {
    if (event_ != nullptr) {
      cudaEventSynchronize(event_);
      cudaEventDestroy(event_);
    }
    if (word_ != nullptr) cudaFreeHost(word_);
  }
  StatusCopy(const StatusCopy&) = delete;
  void start(const Tensor& word) {
    const c10::cuda::CUDAGuard guard(device_);
    const cudaStream_t st = (cudaStream_t)stream_of(word);
    if (cudaMemcpyAsync(word_, word.data_ptr(), sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaEventRecord(event_, st) != cudaSuccess)
      throw Error("status poll: the copy could not be issued");
  }
  // An error of the device is not "still in flight": it is reported here
  bool landed() const {
    const cudaError_t rc = cudaEventQuery(event_);
    if (rc == cudaSuccess) return true;
    cudaGetLastError();   // "not ready" must not be taken for the failure of a later launch
    if (rc != cudaErrorNotReady) throw Error(std::string("status poll: ") + cudaGetErrorString(rc));
    return false;
  }
  int32_t value() const { return *word_; }

 private:
  c10::Device device_;
  int32_t* word_ = nullptr;
  cudaEvent_t event_ = nullptr;
};

void bind_status(pybind11::module_& m) {
  namespace py = pybind11;
  // Has a native backward launched kernels since `clear` was last asked for?
  m.def("backward_ran", [](int64_t device, bool clear) {
    auto& ran = g_backward_ran[device];
    return clear ? ran.exchange(false, std::memory_order_acq_rel) : ran.load(std::memory_order_acquire);
  });
  py::class_<StatusCopy>(m, "StatusCopy")
      .def(py::init<const Tensor&>())
      .def("start", &StatusCopy::start)
      .def("landed", &StatusCopy::landed)
      .def("value", &StatusCopy::value);
}

}  // namespace nsa_host
