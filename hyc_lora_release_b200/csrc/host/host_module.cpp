#include "host.h"

PYBIND11_MODULE(_hyc_host, m) {
  using namespace hyc_host;
  static pybind11::exception<Error> error(m, "HycError", PyExc_RuntimeError);
  pybind11::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const Error& e) {
      PyErr_SetString(error.ptr(), e.what());
    } catch (const c10::ValueError& e) {
      PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
    } catch (const c10::IndexError& e) {
      PyErr_SetString(PyExc_IndexError, e.what_without_backtrace());
    } catch (const c10::OutOfMemoryError& e) {
      PyErr_SetString(pybind11::module_::import("torch").attr("OutOfMemoryError").ptr(), e.what_without_backtrace());
    } catch (const c10::Error& e) {
      PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    }
  });
  bind_ops(m);
  bind_blocks(m);
}
