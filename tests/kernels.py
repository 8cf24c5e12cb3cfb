"""Which kernels a runtime launched (needs the device library): a runtime
with the parameter time_kernel=* times every launch by name."""
import ctypes as C
import json

from equelle_b200.runtime import Runtime


def launched(lib, params, program):
    """program(runtime)'s result, and the names of the kernels it launched."""
    er = Runtime(lib, dict(params, time_kernel="*"))
    out = program(er)
    need = C.c_int64()
    er._ok(lib.eqg_runtime_kernel_profile(er.h, None, 0, C.byref(need)))
    buf = C.create_string_buffer(need.value)
    er._ok(lib.eqg_runtime_kernel_profile(er.h, buf, need.value, C.byref(need)))
    return out, set(json.loads(buf.value.decode()))
