// What the call module (okf_pycall.c) asks of torch, without a Python call: a tensor's address and element type, and the current
// stream.  By method and attribute look-ups these were 250 of the 550 ns that a call took the host before it reached the library; a decode
// step of a small model is 30 to 70 calls.  Only plain tensors are answered for: subclasses, and tensors that have no address (of a
// transform, say), take the look-ups, which raise what torch raises.  A library of its own, named after the torch whose headers it was compiled with: what
// is inlined here (where a tensor keeps its address) holds for that one only, and a torch without CUDA has nothing to link it against.
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/okf_cuda.h"

#define EXPORT extern "C" __attribute__((visibility("default")))

// 1 and the address / okf_dtype; 0: not for this function
EXPORT int okf_tensor_address(PyObject *o, void **out) {
    if (!THPVariable_CheckExact(o)) return 0;
    try {
        *out = THPVariable_Unpack(o).data_ptr();
        return 1;
    } catch (...) {
        return 0;
    }
}
EXPORT int okf_tensor_dtype(PyObject *o, int *out) {
    if (!THPVariable_CheckExact(o)) return 0;
    try {
        switch (THPVariable_Unpack(o).scalar_type()) {
        case at::kFloat: *out = OKF_F32; return 1;
        case at::kHalf: *out = OKF_F16; return 1;
        case at::kBFloat16: *out = OKF_BF16; return 1;
        default: return 0;
        }
    } catch (...) {
        return 0;
    }
}
// 1 and the stream that is current on the current device; 0: ask torch from Python
EXPORT int okf_current_stream(void **out) {
    try {
        *out = c10::cuda::getCurrentCUDAStream().stream();
        return 1;
    } catch (...) {
        return 0;
    }
}
