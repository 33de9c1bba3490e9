// The host extension vmamba_b200/_host.so: module table and error translation.
#include "host_common.h"

namespace host {
void bind_ops(pybind11::module_& m);
void bind_core(pybind11::module_& m);
void bind_backbone(pybind11::module_& m);
}  // namespace host

PYBIND11_MODULE(_host, m) {
    namespace py = pybind11;
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const host::LibError& e) {
            py::object cls = py::module_::import("vmamba_b200._lib").attr("Ss2dError");
            py::object exc = cls(e.status, e.where);
            PyErr_SetObject(cls.ptr(), exc.ptr());
        }
    });
    host::bind_ops(m);
    host::bind_core(m);
    host::bind_backbone(m);
}
