// The Python module of the native host side.

#include <torch/csrc/Exceptions.h>

#include "nsa_host.h"

namespace py = pybind11;

static PyObject* g_error_class = nullptr;   // the package's NsaError, handed over once at load time

static PyObject* error_class() { return g_error_class != nullptr ? g_error_class : PyExc_RuntimeError; }

void nsa_host::raise_python_error(const char* what) {
  const py::gil_scoped_acquire gil;
  PyErr_SetString(error_class(), what);
  python_error err;
  err.persist();
  throw err;
}

PYBIND11_MODULE(_nsa_host, m) {
  m.def("set_error_class", [](py::object cls) { g_error_class = cls.release().ptr(); });
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const nsa_host::Error& e) {
      PyErr_SetString(error_class(), e.what());
    }
  });
  nsa_host::bind_status(m);
  nsa_host::bind_selected(m);
  nsa_host::bind_decode(m);
  nsa_host::bind_layer(m);
}
