// The module nha_b200._nha_host.
#include "nha_host.h"

namespace nha_host {

PyObject* library_error = PyExc_RuntimeError;

static PyObject* set_error(PyObject*, PyObject* type) {
  Py_INCREF(type);
  library_error = type;
  Py_RETURN_NONE;
}

#define NHA_ENTRY(name_) {#name_, (PyCFunction)(void (*)(void))name_, METH_FASTCALL, nullptr}
static PyMethodDef methods[] = {NHA_ENTRY(decode), NHA_ENTRY(decode_logits), NHA_ENTRY(decode_ring),
                                {"decode_workspace", (PyCFunction)(void (*)(void))decode_workspace_for, METH_FASTCALL, nullptr}, NHA_ENTRY(chunk_nha),
                                NHA_ENTRY(prefill), NHA_ENTRY(slot_gates), NHA_ENTRY(rotary_pair), NHA_ENTRY(feature_maps),
                                NHA_ENTRY(silu_rms_norm), NHA_ENTRY(gsa_aux_loss), {"set_error", set_error, METH_O, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nha_host", "Host side of nha_b200's operators.", -1, methods,
                             nullptr, nullptr, nullptr, nullptr};

}  // namespace nha_host

PyMODINIT_FUNC PyInit__nha_host(void) { return PyModule_Create(&nha_host::module); }
