// A copy of a device status word on its way to the host: started after some call, looked at during a later one.

#include <cuda_runtime_api.h>

#include "nsa_host.h"

namespace nsa_host {

class StatusCopy {
 public:
  StatusCopy() {
    if (cudaHostAlloc(reinterpret_cast<void**>(&word_), sizeof(int32_t), cudaHostAllocDefault) != cudaSuccess ||
        cudaEventCreateWithFlags(&event_, cudaEventDisableTiming) != cudaSuccess)
      throw Error("status poll: no pinned word or event");
    *word_ = 0;
  }
  ~StatusCopy() {
    cudaEventSynchronize(event_);
    cudaEventDestroy(event_);
    cudaFreeHost(word_);
  }
  StatusCopy(const StatusCopy&) = delete;
  void start(const Tensor& word) {
    const cudaStream_t st = (cudaStream_t)stream_of(word);
    if (cudaMemcpyAsync(word_, word.data_ptr(), sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaEventRecord(event_, st) != cudaSuccess)
      throw Error("status poll: the copy could not be issued");
  }
  bool landed() const { return cudaEventQuery(event_) == cudaSuccess; }
  int32_t value() const { return *word_; }

 private:
  int32_t* word_ = nullptr;
  cudaEvent_t event_ = nullptr;
};

void bind_status(pybind11::module_& m) {
  namespace py = pybind11;
  py::class_<StatusCopy>(m, "StatusCopy")
      .def(py::init<>())
      .def("start", &StatusCopy::start)
      .def("landed", &StatusCopy::landed)
      .def("value", &StatusCopy::value);
}

}  // namespace nsa_host
