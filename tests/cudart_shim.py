"""A stand-in in front of the CUDA runtime, for tests of the host side: it
notes the kernels launched and the function attributes set, and can refuse one
launch with an error code.  A test runs its program under it in a process of
its own (LD_PRELOAD), as the library is linked against the shared runtime."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>

static void* real(const char* name) {
    static void* rt;
    if (!rt) rt = dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY);
    return dlsym(rt, name);
}

enum { kLog = 1 << 16 };
const void* shim_launched[kLog];   /* host functions of the kernels, in order */
int shim_n_launched;
const void* shim_attr_func[kLog];  /* cudaFuncSetAttribute calls, in order */
int shim_attr[kLog], shim_attr_value[kLog];
int shim_n_attr;
int shim_refuse = -1;              /* launches to let pass before one is refused (-1: none) */
int shim_refuse_captured;          /* which ones count: 0 launches with attributes, not captured; 1 captured ones */
static cudaError_t pending;

static int refuse(cudaStream_t s, int attributes) {
    enum cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (shim_refuse < 0) return 0;
    ((cudaError_t(*)(cudaStream_t, enum cudaStreamCaptureStatus*))real("cudaStreamIsCapturing"))(s, &st);
    if (shim_refuse_captured ? st != cudaStreamCaptureStatusActive : st == cudaStreamCaptureStatusActive || !attributes)
        return 0;
    if (shim_refuse-- > 0) return 0;
    pending = cudaErrorInvalidConfiguration;
    return 1;
}
static void note(const void* f) {
    if (shim_n_launched < kLog) shim_launched[shim_n_launched++] = f;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t m, cudaStream_t s) {
    note(f);
    if (refuse(s, 0)) return pending;
    return ((cudaError_t(*)(const void*, dim3, dim3, void**, size_t, cudaStream_t))real("cudaLaunchKernel"))(f, g, b, a, m, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
    note(f);
    if (refuse(c->stream, 1)) return pending;
    return ((cudaError_t(*)(const cudaLaunchConfig_t*, const void*, void**))real("cudaLaunchKernelExC"))(c, f, a);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute k, int v) {
    if (shim_n_attr < kLog) {
        shim_attr_func[shim_n_attr] = f;
        shim_attr[shim_n_attr] = (int)k;
        shim_attr_value[shim_n_attr++] = v;
    }
    return ((cudaError_t(*)(const void*, enum cudaFuncAttribute, int))real("cudaFuncSetAttribute"))(f, k, v);
}
/* a refused launch is the last error, as a real one is, until it is asked for */
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = pending;
    pending = cudaSuccess;
    if (e != cudaSuccess) return e;
    return ((cudaError_t(*)(void))real("cudaGetLastError"))();
}
"""

# what every program starts with: the shim's variables by name, and the kernels that some calls launch
PRELUDE = r"""
import ctypes as C, os, sys
sys.path.insert(0, %r)
import numpy as np
import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE
shim = C.CDLL(os.environ["LD_PRELOAD"])
def var(name, kind=C.c_int):
    return kind.in_dll(shim, name)
def kernels(call):
    first = var("shim_n_launched").value
    call()
    return list(var("shim_launched", C.c_void_p * 65536)[first:var("shim_n_launched").value])
""" % ROOT


def run(tmp_path, program, timeout=300):
    """Runs `program` (after PRELUDE) under the shim; what it printed."""
    so = os.path.join(str(tmp_path), "cudart_shim.so")
    src = os.path.join(str(tmp_path), "cudart_shim.c")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", src, "-o", so, "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", PRELUDE + program], env=dict(os.environ, LD_PRELOAD=so), timeout=timeout,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
